// kaczmarz.cu -- the ordered row-action sweep of basic_sweep
// (AIRMs.f90:813-858) on the GPU.
//
// The sweep is strictly sequential (adjacent rays share pixels), so one
// thread block walks the reference's row order; its W warps share each row's
// dot product (csr_matrowvec, sparse_matrices.f90:252-270) and bounded update
// (add_mult_row, :795-822). Row k+1 starts only after row k's update is
// visible, so the iterate follows the reference's sequence of projections.
// Three roundings differ from the reference: a_i.x - b_i is exact before its
// one rounding (the reference rounds each term of its ordered sum), the
// update is one fused multiply-add, and the coefficient is formed as
// (b_i - a_i.x) * (omega / nrA_i) instead of omega * (b_i - a_i.x) / nrA_i
// (AIRMs.f90:842).
//
// On GB300 every FP64 warp instruction holds its SM sub-partition's FP64 pipe
// for 64 cycles (measured: a dependent and an independent chain of DFMA both
// issue one per 64 cycles per warp), whatever its active lanes, and a
// row-action sweep runs on one SM; a row is a dependent chain (dot product,
// reduction, coefficient, update). The kernel therefore spends FP64
// instructions only where the arithmetic needs them:
//  * a row's entries are spread densely over the block (len / (32 W)
//    instructions per lane, skipped by a block-uniform branch past the end);
//  * the row sum a_i.x - b_i is formed exactly on the integer pipes (the
//    lanes' partials as 64-bit fixed point in a common frame, added by warp
//    reductions) and rounded once, so the reduction tree and the subtraction
//    of b_i use no FP64 instruction; each warp adds the W warp sums itself,
//    so one barrier per row suffices;
//  * omega / nrA_i, b_i and each step's entry range come from a parallel
//    schedule kernel, together with the row sampled by row probability
//    (AIRMs.f90:830-835);
//  * the box constraints are applied with integer comparisons on an
//    order-preserving key of the IEEE bits (the gfortran MAX/MIN semantics:
//    a NaN operand loses, +0 and -0 compare equal).
// The step record two rows ahead and the next row's column indices and
// values are prefetched while the current row is worked on, and the gathered
// values of x stay in registers for the update.
//
// When the iterate fits in shared memory it is kept there for the whole
// sweep; otherwise it stays in global memory (L2-resident at these sizes).
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>

#include "fair_internal.cuh"
#include "grid_barrier.cuh"

namespace fair {

namespace {

struct RowStep {
    int64_t s;    // first entry of the row
    int32_t len;  // entries
    int32_t level;  // in a level schedule: the step's level
    double b;     // b(ri)
    double w;     // omega / nrA(ri)
};

// first index i in [0, m) with cumul[i] >= u (the linear scan of
// AIRMs.f90:831-835 finds the same row on the nondecreasing cumul); m-1 if none
__device__ __forceinline__ int32_t sample_row(const double *cumul, int32_t m, double u) {
    int32_t L = 0, R = m;
    while (L < R) {
        int32_t mid = (L + R) >> 1;
        if (__ldg(cumul + mid) >= u) R = mid; else L = mid + 1;
    }
    return L < m ? L : m - 1;
}

__global__ void k_sweep_schedule(const int32_t *ord, int32_t nord, int dir, int rowprob,
                                 const double *cumul, int32_t m, uint64_t seed, uint64_t ctr,
                                 const int64_t *rowptr, const double *b, const double *nrA,
                                 double omg, RowStep *steps) {
    for (int32_t ii = blockIdx.x * blockDim.x + threadIdx.x; ii < nord;
         ii += gridDim.x * blockDim.x) {
        int32_t ri = rowprob ? sample_row(cumul, m, uniform01(seed, ctr + (uint64_t)ii))
                             : ord[dir > 0 ? ii : nord - 1 - ii] - 1;
        int64_t s = rowptr[ri];
        steps[ii] = RowStep{s, (int32_t)(rowptr[ri + 1] - s), 0, b[ri], __ddiv_rn(omg, nrA[ri])};
    }
}

// Order-preserving key of a non-NaN double: key(-x) = -key(x), key(+-0) = 0.
__host__ __device__ __forceinline__ long long okey(long long bits) {
    long long mag = bits & 0x7FFFFFFFFFFFFFFFLL;
    return bits < 0 ? -mag : mag;
}
__device__ __forceinline__ bool is_nan_bits(long long bits) {
    return (bits & 0x7FFFFFFFFFFFFFFFLL) > 0x7FF0000000000000LL;
}

struct Box {
    int mode;  // bit0: upper bound, bit1: lower bound
    long long klb, kub;
    double lb, ub;
    // add_mult_row (sparse_matrices.f90:812-818): MAX(t, lb) first, then
    // MIN(t, ub); MAX/MIN return the non-NaN operand
    __device__ __forceinline__ double apply(double t) const {
        if (mode & 2) {
            long long tb = __double_as_longlong(t);
            if (klb > okey(tb) || is_nan_bits(tb)) t = lb;
        }
        if (mode & 1) {
            long long tb = __double_as_longlong(t);
            if (kub < okey(tb) || is_nan_bits(tb)) t = ub;
        }
        return t;
    }
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// ---- exact sums of doubles on the integer pipes ------------------------------
// A finite double with exponent field e and significand m (53 bits with the
// implicit one; e = 0: no implicit one, scale as e = 1) is m * 2^(e - 1075).
// In the frame E (at least every term's e) it becomes the integer m >> (E - e),
// which drops less than one unit 2^(E - 1075): an ulp of the largest term. A
// warp adds its lanes' integers exactly as three 26-bit limbs with
// __reduce_add_sync, the warps' sums are aligned to the largest frame, and the
// total is rounded to double once (round to nearest even). A row of up to
// 8 x 32 lanes x 2 partials + b stays below 2^63; 16 warps' may not (fx_group).
__device__ __forceinline__ int fx_exp(double v) {
    const int e = (int)((__double_as_longlong(v) >> 52) & 0x7FF);
    return e > 1 ? e : 1;
}
__device__ __forceinline__ long long fx_of(double v, int E) {
    const long long b = __double_as_longlong(v);
    const int e = (int)((b >> 52) & 0x7FF);
    long long m = b & 0xFFFFFFFFFFFFFLL;
    if (e) m |= 1LL << 52;
    const int sh = E - (e > 1 ? e : 1);
    const long long f = sh < 64 ? (m >> sh) : 0LL;
    return b < 0 ? -f : f;
}
__device__ __forceinline__ long long fx_warp_sum(long long F) {  // |F| < 2^60 per lane
    const unsigned l0 = __reduce_add_sync(0xffffffffu, (unsigned)(F & 0x3FFFFFF));
    const unsigned l1 = __reduce_add_sync(0xffffffffu, (unsigned)((F >> 26) & 0x3FFFFFF));
    const int l2 = __reduce_add_sync(0xffffffffu, (int)(F >> 52));
    return (long long)l2 * (1LL << 52) + (long long)l1 * (1LL << 26) + (long long)l0;
}
// total * 2^(E - 1075) rounded to nearest even, once. Below the normal range
// the value is exact: the frame's unit 2^(E - 1075) (E >= 1) is a multiple of
// the smallest subnormal 2^-1074, and such a total has fewer than 53 - E + 1
// bits, so it is the subnormal significand shifted by E - 1. Above it the
// rounded value overflows to infinity.
__device__ __forceinline__ double fx_to_double(long long total, int E) {
    if (total == 0) return 0.0;
    const bool neg = total < 0;
    unsigned long long a = neg ? 0ull - (unsigned long long)total : (unsigned long long)total;
    int nb = 64 - __clzll((long long)a);
    unsigned long long mant;
    if (nb <= 53) {
        mant = a << (53 - nb);
    } else {
        const int sh = nb - 53;
        mant = a >> sh;
        const unsigned long long rem = a & ((1ull << sh) - 1ull), half = 1ull << (sh - 1);
        if (rem > half || (rem == half && (mant & 1ull))) ++mant;
        if (mant == (1ull << 53)) {
            mant >>= 1;
            ++nb;
        }
    }
    const int field = nb + E - 53;
    unsigned long long bits;
    if (field < 1) bits = a << (E - 1);  // nb <= 53 - E here: no rounding above, < 2^52
    else if (field > 2046) bits = 0x7FF0000000000000ull;
    else bits = ((unsigned long long)field << 52) | (mant & 0xFFFFFFFFFFFFFull);
    if (neg) bits |= 1ull << 63;
    return __longlong_as_double((long long)bits);
}
// A warp's share of a row sum: its integer sum in its frame, or (when a term
// is Inf or NaN, frame 0x7FF) its FP64 sum.
struct FxPart {
    long long s;
    double d;
    int e;
    int pad;
};
__device__ __forceinline__ FxPart fx_warp_part(double p0, double p1, double p2) {
    int e = max(max(fx_exp(p0), fx_exp(p1)), fx_exp(p2));
    FxPart r{0, 0.0, (int)__reduce_max_sync(0xffffffffu, (unsigned)e), 0};
    if (r.e < 0x7FF) r.s = fx_warp_sum(fx_of(p0, r.e) + fx_of(p1, r.e) + fx_of(p2, r.e));
    else r.d = warp_sum(p0 + p1 + p2);
    return r;
}
// The row sum from the warps' shares (FP64 sum of the non-finite shares when
// there are any: an Inf or NaN term decides the result).
template <int W>
__device__ __forceinline__ double fx_total(const FxPart *part) {
    int E = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) E = max(E, part[w].e);
    if (E >= 0x7FF) {
        double d = 0.0;
#pragma unroll
        for (int w = 0; w < W; ++w)
            if (part[w].e >= 0x7FF) d += part[w].d;
        return d;
    }
    long long t = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) {
        const int sh = E - part[w].e;
        if (sh < 64) t += part[w].s >> sh;
    }
    return fx_to_double(t, E);
}

// dup: when given and set, some row repeats a column (found by the level
// set-up); thread 0 then applies each row's updates one entry after the other,
// so that a repeated column takes both updates in order as in add_mult_row.
// only_if_dup: the level sweep ran; this kernel runs only for such a matrix.
template <int W, int CACHE, bool SMEM_X>
__global__ void __launch_bounds__(32 * W) k_sweep(const RowStep *__restrict__ steps, int32_t nord,
                                                  const int32_t *__restrict__ col,
                                                  const double *__restrict__ val, double *xg,
                                                  int32_t n, Box box, const int *dup,
                                                  int only_if_dup) {
    constexpr int T = 32 * W;
    extern __shared__ double xs[];
    __shared__ FxPart part_s[W];
    const bool serial_update = dup && *dup;
    if (only_if_dup && !serial_update) return;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    double *x = SMEM_X ? xs : xg;
    if (SMEM_X) {
        for (int32_t j = tid; j < n; j += T) xs[j] = xg[j];
        __syncthreads();
    }
    if (nord <= 0) return;
    const RowStep none{0, 0, 0, 0.0, 0.0};
    // three-stage pipeline: the step record two rows ahead, the entries of
    // the next row, the current row
    RowStep cur = steps[0];
    RowStep nxt = nord > 1 ? steps[1] : none;
    int32_t cc[CACHE];
    double vv[CACHE];
    int nq = (cur.len + T - 1) / T;
#pragma unroll
    for (int q = 0; q < CACHE; ++q) {
        if (q >= nq) break;
        int k = tid + q * T;
        cc[q] = k < cur.len ? __ldg(col + cur.s + k) : 0;
        vv[q] = k < cur.len ? __ldg(val + cur.s + k) : 0.0;
    }
    for (int32_t ii = 0; ii < nord; ++ii) {
        const RowStep nxt2 = ii + 2 < nord ? steps[ii + 2] : none;
        const int nqn = (nxt.len + T - 1) / T;
        int32_t nc[CACHE];
        double nv[CACHE];
#pragma unroll
        for (int q = 0; q < CACHE; ++q) {
            if (q >= nqn) break;
            int k = tid + q * T;
            nc[q] = k < nxt.len ? __ldg(col + nxt.s + k) : 0;
            nv[q] = k < nxt.len ? __ldg(val + nxt.s + k) : 0.0;
        }
        // dot product of the row with x (two independent accumulators)
        double xo[CACHE];
        double p0 = 0.0, p1 = 0.0;
#pragma unroll
        for (int q = 0; q < CACHE; ++q) {
            if (q >= nq) break;
            int k = tid + q * T;
            xo[q] = k < cur.len ? x[cc[q]] : 0.0;
        }
#pragma unroll
        for (int q = 0; q < CACHE; ++q) {
            if (q >= nq) break;
            if (q & 1) p1 = fma(xo[q], vv[q], p1); else p0 = fma(xo[q], vv[q], p0);
        }
        for (int k = tid + CACHE * T; k < cur.len; k += T)
            p0 = fma(x[__ldg(col + cur.s + k)], __ldg(val + cur.s + k), p0);
        // a_i.x - b_i, summed exactly on the integer pipes (-b_i is a term of
        // thread 0) and rounded once; every warp forms the same total, so the
        // coefficient needs no second barrier
        const FxPart mine = fx_warp_part(p0, p1, tid == 0 ? -cur.b : 0.0);
        double resid;
        if (W > 1) {
            if (lane == 0) part_s[wid] = mine;
            __syncthreads();
            resid = fx_total<W>(part_s);
        } else {
            resid = fx_total<1>(&mine);
        }
        const double coeff = __dmul_rn(-resid, cur.w);
        if (serial_update) {
            // every thread's reads of x for this row are done (the barrier above,
            // or the warp's reductions)
            if (tid == 0)
                for (int k = 0; k < cur.len; ++k) {
                    const int32_t c = __ldg(col + cur.s + k);
                    x[c] = box.apply(fma(coeff, __ldg(val + cur.s + k), x[c]));
                }
        } else {
#pragma unroll
            for (int q = 0; q < CACHE; ++q) {
                if (q >= nq) break;
                int k = tid + q * T;
                if (k < cur.len) x[cc[q]] = box.apply(fma(coeff, vv[q], xo[q]));
            }
            for (int k = tid + CACHE * T; k < cur.len; k += T) {
                int32_t c = __ldg(col + cur.s + k);
                x[c] = box.apply(fma(coeff, __ldg(val + cur.s + k), x[c]));
            }
        }
        if (W > 1) __syncthreads(); else __syncwarp();
        cur = nxt;
        nxt = nxt2;
        nq = nqn;
#pragma unroll
        for (int q = 0; q < CACHE; ++q) { cc[q] = nc[q]; vv[q] = nv[q]; }
    }
    if (SMEM_X) {
        __syncthreads();
        for (int32_t j = tid; j < n; j += T) xg[j] = xs[j];
    }
}

template <int W, int CACHE>
int launch(const SweepDev &S, const RowStep *steps, bool smem, size_t smem_bytes, const Box &box,
           const int *dup, int only_if_dup, cudaStream_t s) {
    const DevCSR &A = *S.A;
    if (smem) {
        auto kern = k_sweep<W, CACHE, true>;
        FAIR_CUDA(smem_allow(reinterpret_cast<const void *>(kern), smem_bytes));
        kern<<<1, 32 * W, smem_bytes, s>>>(steps, S.nord, A.col.as<int32_t>(), A.v64.as<double>(),
                                          S.x, A.n, box, dup, only_if_dup);
    } else {
        k_sweep<W, CACHE, false><<<1, 32 * W, 0, s>>>(steps, S.nord, A.col.as<int32_t>(),
                                                     A.v64.as<double>(), S.x, A.n, box, dup,
                                                     only_if_dup);
    }
    FAIR_CUDA(cudaGetLastError());
    return FAIR_OK;
}

long long host_key(double v) {
    long long bits;
    memcpy(&bits, &v, sizeof bits);
    return okey(bits);
}

// Warps per row: FAIR_SWEEP_WARPS (1, 2, 4 or 8) when set, else 4. Measured
// on GB300 (host call, rows/s for 1, 2, 4, 8 warps): fan beam N=128, x in
// shared memory, Kaczmarz 0.83M, 0.97M, 1.00M, 0.94M; fan beam N=512, x in
// global memory, symmetric Kaczmarz 0.18M, 0.33M, 0.44M, 0.39M and random
// Kaczmarz 0.17M, 0.30M, 0.43M, 0.42M.
int sweep_warps() {
    const char *env = getenv("FAIR_SWEEP_WARPS");
    if (env) {
        int w = atoi(env);
        if (w == 1 || w == 2 || w == 4 || w == 8) return w;
    }
    return 4;
}

// ---- level-scheduled sweep ------------------------------------------------------
// Two steps of a sweep commute when their rows share no column: neither reads
// what the other writes. Give step k the level 1 + max(level of every earlier
// step sharing a column with it); then every step's reads come after all
// earlier steps that write those columns and before all later ones, so running
// the levels in order, the steps of one level in parallel, gives exactly the
// sequence of bounded projections of basic_sweep (AIRMs.f90:813-858): the
// same row sums (exact fixed-point sums of the lanes' FP64 partials, rounded
// once) and the same updates in the same order per column. For a ray order
// that walks the bins of one angle and then the next, the levels form a
// wavefront: a ray waits for its neighbour bin and for the few rays of the
// previous angle that cross its pixels, so about 30 (fan beam N=128) to 80
// (N=512) steps share a level.
//
// The levels are exact, computed per sweep order in windows of WR = 128 steps
// (64 or 32 where a window's entries would not fit shared memory):
//   k_lvl_setup (every SM, windows in parallel): each entry swaps a stamp
//     into its column's cell of the block's table; a stamp of an earlier step
//     of the window makes the entry "shared" and that step a predecessor; the
//     step's entries are written in groups [first touch in the window and
//     last | first, not last | shared, not last | shared and last], and the
//     longest paths between the window's steps (predecessor chains) as one
//     byte per pair;
//   k_lvl_levels_grid (a step of the window per block of a cooperative grid; where
//     that launch is refused k_lvl_levels_cluster, on a 16-block cluster, or
//     k_lvl_levels, in one block), windows in order: a step's level
//     is the largest, over the steps a of its window with a path to it, of
//     base(a) + the path's length, base(a) = 1 + the table's level over a's
//     first-touch columns; the last touches write the levels into the table
//     (a window costs two rounds of scattered table accesses and the exchanges
//     between them whatever it holds: fan N=512, 243,328 steps, on a cluster
//     32.5 ms in windows of 32, 13.9 ms in windows of 128);
//   counting sort of the steps by level (level pointers, steps in level order).
// The sweep in the direction the levels were built for runs without barriers
// (k_flow_sweep): every x_j carries the level that updated it last, and a step
// waits for its own columns only. The opposite direction takes the levels in
// reverse (k_lvl_sweep): a group of G warps per step, the steps of a
// level spread over the groups, on one thread-block cluster (a cluster barrier
// between levels; x in the cluster's distributed shared memory when its parts
// fit, else in global memory read past L1) or, when a level outgrows the
// cluster, on a cooperative grid of up to one block per SM (a software grid
// barrier between levels; x in global memory); so does a sweep for whose copies
// of the entries there is no memory.

struct WinRow {
    int64_t off;              // first entry of the step in the grouped column array
    int32_t len, c1, c2, c3;  // entries; groups [0,c1) [c1,c2) [c2,c3) [c3,len)
};
static_assert(sizeof(WinRow) == 24, "WinRow layout");

constexpr int kMinStepsPerLevel = 4;
constexpr int kSetupThreads = 512;
constexpr int kSetupWarps = kSetupThreads / 32;
// Window stamps of the set-up's column tables: window id (36 bits), step in
// the window (8 bits), entry position in the window (20 bits). All ones marks
// an empty cell.
constexpr int kStampPosBits = 20;
constexpr unsigned long long kStampIdLimit = (1ull << 36) - 1ull;

__device__ __forceinline__ unsigned long long win_stamp(unsigned long long id, int r, int pos) {
    return (id << 28) | ((unsigned long long)r << kStampPosBits) | (unsigned long long)pos;
}
// group of an entry from its flags (bit 0: a later step of the window has the
// column; bits 1-7: 1 + the last earlier step that has it, 0: none)
__device__ __forceinline__ int win_group(unsigned f) {
    return f > 1u ? ((f & 1u) ? 2 : 3) : (int)f;
}

// total * 2^(E - 1075), rounded once: the integer converted to double (round
// to nearest even) and rescaled by its exponent field when the result is a
// normal number; otherwise fx_to_double.
__device__ __forceinline__ double fx_to_double_fast(long long total, int E) {
    if (total == 0) return 0.0;
    const long long bits = __double_as_longlong(__ll2double_rn(total));
    const int field = (int)((bits >> 52) & 0x7FF) + E - 1075;
    if (field >= 1 && field <= 2046)
        return __longlong_as_double(bits + ((long long)(E - 1075) << 52));
    return fx_to_double(total, E);
}

// The sum of the lanes' aligned parts F (|F| < 2^59 + 2^53), rounded once. 16
// parts can reach 2^63 + 2^53: a total near the ends of 64 bits is formed halved,
// its lost bit kept as the lowest one, which no rounding to 53 bits looks past.
__device__ __forceinline__ double fx_group(long long F, int E) {
    const unsigned l0 = __reduce_add_sync(0xffffffffu, (unsigned)(F & 0x3FFFFFF));
    const unsigned l1 = __reduce_add_sync(0xffffffffu, (unsigned)((F >> 26) & 0x3FFFFFF));
    const int l2 = __reduce_add_sync(0xffffffffu, (int)(F >> 52));
    const long long m = (long long)l1 * (1LL << 26) + (long long)l0;  // < 2^57 + 2^31
    if ((unsigned)(l2 + 2048) < 4096u - 33u) return fx_to_double_fast((long long)l2 * (1LL << 52) + m, E);
    return fx_to_double(((long long)l2 * (1LL << 51) + (m >> 1)) | (m & 1LL), E + 1);
}

// The FP64 sum of the parts that hold an Inf or NaN term.
__device__ __noinline__ double fx_special(const FxPart *parts, int G) {
    double d = 0.0;
    for (int w = 0; w < G; ++w)
        if (parts[w].e >= 0x7FF) d += parts[w].d;
    return d;
}

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\t"
                 "barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

// Exclusive scan of n counts (n from *n_dev when given) into out[0..n], one
// block.
__global__ void __launch_bounds__(1024) k_scan_excl(const int32_t *__restrict__ in, int64_t n_host,
                                                   const int *__restrict__ n_dev,
                                                   int64_t *__restrict__ out) {
    __shared__ int64_t wsum[32];
    __shared__ int64_t carry;
    const int64_t n = n_dev ? (int64_t)*n_dev : n_host;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    if (tid == 0) carry = 0;
    __syncthreads();
    for (int64_t b = 0; b < n; b += 1024) {
        const int64_t i = b + tid;
        int64_t v = i < n ? in[i] : 0, inc = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        if (lane == 31) wsum[wid] = inc;
        __syncthreads();
        if (wid == 0) {
            int64_t w = wsum[lane], wi = w;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int64_t t = __shfl_up_sync(0xffffffffu, wi, o);
                if (lane >= o) wi += t;
            }
            wsum[lane] = wi - w;
        }
        __syncthreads();
        const int64_t c = carry;
        if (i < n) out[i] = c + wsum[wid] + inc - v;
        __syncthreads();
        if (tid == 1023) carry = c + wsum[31] + inc;
        __syncthreads();
    }
    if (tid == 0) out[n] = carry;
}

__global__ void k_step_lengths(const RowStep *__restrict__ steps, int32_t nord,
                               int32_t *__restrict__ lens) {
    for (int32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < nord; k += gridDim.x * blockDim.x)
        lens[k] = steps[k].len;
}

// Set-up of the windows (one block per window at a time, a table per block).
// The steps of a window are taken in order; each entry swaps its stamp into
// its column's cell, and the stamp it finds tells whether an earlier step of
// the window has the column (this entry is then shared, that one not last,
// and that step a predecessor of this one). A stamp of the same step means the
// row repeats a column: *err is set and the single-block kernel applies the
// sweep's updates in order instead. From the predecessors, the longest path
// between every two steps of the window (dpath: a byte per pair). Bound by the
// round trip of a step's swaps, step by step; the next step's columns are
// loaded meanwhile (fan N=512: 6.1 -> 4.7 ms, N=128 0.27 -> 0.19 ms).
template <int WR>
__global__ void __launch_bounds__(kSetupThreads) k_lvl_setup(
        const RowStep *__restrict__ steps, const int64_t *__restrict__ eoff, int32_t nord,
        const int32_t *__restrict__ col, unsigned long long *__restrict__ tabs, int32_t n,
        unsigned long long id0, int32_t *__restrict__ oidx, WinRow *__restrict__ rec,
        unsigned char *__restrict__ dpath, const double *__restrict__ val, double *__restrict__ oval,
        int32_t *__restrict__ otag, int *err) {
    extern __shared__ __align__(16) unsigned char fl[];  // [entries of a window]
    __shared__ int rb[WR + 1];
    __shared__ int64_t rs[WR];             // first entries of the rows
    __shared__ uint32_t msk[WR][WR / 32];  // predecessor steps in the window
    __shared__ uint32_t dps[WR][WR / 4];   // 1 + longest path a -> r, 0: none (a byte per a)
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    unsigned long long *tab = tabs + (size_t)blockIdx.x * (size_t)n;
    const int nwin = (nord + WR - 1) / WR;
    for (int q = blockIdx.x; q < nwin; q += gridDim.x) {
        const int k0 = q * WR, nr = min(WR, nord - k0);
        const int64_t wbase = eoff[k0];
        if (tid < WR) {
            rb[tid + 1] = tid < nr ? (int)(eoff[k0 + tid + 1] - wbase) : 0;
            rs[tid] = tid < nr ? steps[k0 + tid].s : 0;
            for (int w = 0; w < WR / 32; ++w) msk[tid][w] = 0;
            if (tid == 0) rb[0] = 0;
        }
        __syncthreads();
        const unsigned long long id = id0 + (unsigned long long)q;
        // the columns of the next row are on their way during a row's swaps
        constexpr int JC = 2;  // columns per thread in registers
        int32_t cj[JC];
        auto fetch = [&](int r) {
            const int64_t s0 = r < nr ? rs[r] : 0;
            const int len = r < nr ? rb[r + 1] - rb[r] : 0;
#pragma unroll
            for (int t = 0; t < JC; ++t)
                cj[t] = tid + kSetupThreads * t < len ? __ldg(col + s0 + tid + kSetupThreads * t) : -1;
        };
        fetch(0);
        for (int r = 0; r < nr; ++r) {
            const int base = rb[r], len = rb[r + 1] - base;
            auto swap = [&](int e, int32_t c) {
                const int pos = base + e;
                const unsigned long long old = atomicExch(tab + c, win_stamp(id, r, pos));
                unsigned char f = 0;
                if ((old >> 28) == id) {
                    const int orow = (int)((old >> kStampPosBits) & 0xFFull);
                    if (orow == r) {
                        atomicExch(err, 1);
                    } else {
                        f = (unsigned char)((orow + 1) << 1);
                        fl[old & ((1ull << kStampPosBits) - 1ull)] |= 1;  // its one writer
                        atomicOr(&msk[r][orow >> 5], 1u << (orow & 31));
                    }
                }
                fl[pos] = f;
            };
            int32_t c[JC];
#pragma unroll
            for (int t = 0; t < JC; ++t) c[t] = cj[t];
            fetch(r + 1);
#pragma unroll
            for (int t = 0; t < JC; ++t)
                if (c[t] >= 0) swap(tid + kSetupThreads * t, c[t]);
            for (int e = tid + kSetupThreads * JC; e < len; e += kSetupThreads) swap(e, col[rs[r] + e]);
            __syncthreads();
        }
        if (wid == 0 && lane < WR / 4) {  // longest paths within the window (rows in order),
                                          // four steps a per lane
            constexpr unsigned LANES = WR / 4 == 32 ? 0xffffffffu : (1u << (WR / 4)) - 1u;
            for (int r = 0; r < nr; ++r) {
                uint32_t v = lane == r >> 2 ? 1u << (8 * (r & 3)) : 0u;
#pragma unroll
                for (int w = 0; w < WR / 32; ++w)
                    for (uint32_t bits = msk[r][w]; bits; bits &= bits - 1u) {
                        const uint32_t d = dps[32 * w + __ffs(bits) - 1][lane];
                        v = __vmaxu4(v, __vaddus4(d, 0x01010101u) & __vcmpne4(d, 0u));
                    }
                dps[r][lane] = v;
                __syncwarp(LANES);
            }
            for (int r = 0; r < nr; ++r)
                reinterpret_cast<uint32_t *>(dpath + (size_t)(k0 + r) * WR)[lane] = dps[r][lane];
        }
        const unsigned lt = (1u << lane) - 1u;
        for (int r = wid; r < nr; r += kSetupWarps) {
            const int64_t s0 = steps[k0 + r].s;
            const int base = rb[r], len = rb[r + 1] - base;
            int n0 = 0, n1 = 0, n2 = 0;
            for (int e0 = 0; e0 < len; e0 += 32) {
                const int e = e0 + lane;
                const int g = e < len ? win_group(fl[base + e]) : -1;
                n0 += __popc(__ballot_sync(0xffffffffu, g == 0));
                n1 += __popc(__ballot_sync(0xffffffffu, g == 1));
                n2 += __popc(__ballot_sync(0xffffffffu, g == 2));
            }
            int o0 = 0, o1 = n0, o2 = n0 + n1, o3 = n0 + n1 + n2;
            const int64_t ro = wbase + base;
            for (int e0 = 0; e0 < len; e0 += 32) {
                const int e = e0 + lane;
                const unsigned f = e < len ? fl[base + e] : 0u;
                const int g = e < len ? win_group(f) : -1;
                const unsigned b0 = __ballot_sync(0xffffffffu, g == 0);
                const unsigned b1 = __ballot_sync(0xffffffffu, g == 1);
                const unsigned b2 = __ballot_sync(0xffffffffu, g == 2);
                const unsigned b3 = __ballot_sync(0xffffffffu, g == 3);
                if (g >= 0) {
                    const int d = g == 0 ? o0 + __popc(b0 & lt)
                                : g == 1 ? o1 + __popc(b1 & lt)
                                : g == 2 ? o2 + __popc(b2 & lt)
                                         : o3 + __popc(b3 & lt);
                    oidx[ro + d] = col[s0 + e];
                    if (otag) {
                        oval[ro + d] = val[s0 + e];
                        if (f > 1u) otag[ro + d] = -(int)(f >> 1);  // k_lvl_tags looks the step up
                    }
                }
                o0 += __popc(b0);
                o1 += __popc(b1);
                o2 += __popc(b2);
                o3 += __popc(b3);
            }
            if (lane == 0) rec[k0 + r] = WinRow{ro, len, n0, n0 + n1, n0 + n1 + n2};
        }
        __syncthreads();  // fl, rb, msk and dps belong to the next window
    }
}

// The steps' levels, windows in order (one block of 1024 threads, warp w the
// steps w, w + 32, ... of a window). lv: the last level written into each
// column (shared memory when it fits, else global memory, zeroed by the
// caller). A step's level is the largest, over the steps a of its window with a
// path to it, of base(a) + the path's length, where base(a) = 1 + the table's
// level over a's first-touch columns. The next window's records are loaded
// while a window runs.
template <int WR, bool SMEM>
__global__ void __launch_bounds__(1024, 1) k_lvl_levels(
        const WinRow *__restrict__ rec, const unsigned char *__restrict__ dpath,
        const int32_t *__restrict__ oidx, int32_t nord, int32_t *lvg, int32_t n,
        int32_t *__restrict__ lvl, int32_t *__restrict__ otag, int *__restrict__ nlev) {
    constexpr int SW = WR / 32;  // steps per warp
    extern __shared__ int32_t lvs[];
    __shared__ int32_t base[WR];
    __shared__ int s_top[32];
    int32_t *lv = SMEM ? lvs : lvg;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    if (SMEM)
        for (int32_t j = tid; j < n; j += 1024) lvs[j] = 0;
    const WinRow none{0, 0, 0, 0, 0};
    const int nwin = (nord + WR - 1) / WR;
    WinRow wn[SW];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < SW; ++i) {
            const int k = k0 + wid + 32 * i;
            wn[i] = k < nord ? rec[k] : none;
        }
    };
    fetch(0);
    __syncthreads();
    int top = 0;
    for (int q = 0; q < nwin; ++q) {
        const int k0 = q * WR, nr = min(WR, nord - k0);
        WinRow w[SW];
        uint32_t d[SW];  // dpath of the warp's steps: step a = SW lane + j in byte j
#pragma unroll
        for (int i = 0; i < SW; ++i) {
            w[i] = wn[i];
            const int r = wid + 32 * i;
            d[i] = 0;
            if (r < nr) {
                const unsigned char *p = dpath + (size_t)(k0 + r) * WR + SW * lane;
                if constexpr (SW == 4) d[i] = *reinterpret_cast<const uint32_t *>(p);
                else if constexpr (SW == 2) d[i] = *reinterpret_cast<const uint16_t *>(p);
                else d[i] = *p;
            }
        }
        if (q + 1 < nwin) fetch(k0 + WR);
#pragma unroll
        for (int i = 0; i < SW; ++i) {  // 1 + the table's level over the step's first-touch columns
            const int r = wid + 32 * i;
            if (r >= nr) break;
            int m = 0;
            for (int e0 = lane; e0 < w[i].c2; e0 += 32 * 8) {  // 8 independent loads per lane
                int32_t j[8];
#pragma unroll
                for (int t = 0; t < 8; ++t) j[t] = e0 + 32 * t < w[i].c2 ? oidx[w[i].off + e0 + 32 * t] : -1;
#pragma unroll
                for (int t = 0; t < 8; ++t)
                    if (j[t] >= 0) {
                        const int32_t v = SMEM ? lvs[j[t]] : __ldcg(lvg + j[t]);
                        m = max(m, v);
                        if (otag) otag[w[i].off + e0 + 32 * t] = v;
                    }
            }
            m = (int)__reduce_max_sync(0xffffffffu, (unsigned)m);
            if (lane == 0) base[r] = m + 1;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < SW; ++i) {
            const int r = wid + 32 * i;
            if (r >= nr) break;
            unsigned v = 0;  // the longest path to the step (a path has length d - 1)
#pragma unroll
            for (int j = 0; j < SW; ++j) {
                const unsigned dj = d[i] >> (8 * j) & 255u;
                if (dj > 0) v = max(v, (unsigned)base[SW * lane + j] + dj - 1u);
            }
            const int L = (int)__reduce_max_sync(0xffffffffu, v);
            if (lane == 0) lvl[k0 + r] = L;
            top = max(top, L);
            // the last touches of the window write the step's level
            for (int e0 = lane; e0 < w[i].len; e0 += 32 * 8) {
                int32_t j[8];
#pragma unroll
                for (int t = 0; t < 8; ++t) {
                    const int e = e0 + 32 * t;
                    j[t] = e < w[i].len && (e < w[i].c1 || e >= w[i].c3) ? oidx[w[i].off + e] : -1;
                }
#pragma unroll
                for (int t = 0; t < 8; ++t)
                    if (j[t] >= 0) lv[j[t]] = L;
            }
        }
        __syncthreads();
    }
    if (lane == 0) s_top[wid] = top;
    __syncthreads();
    if (tid == 0) {
        for (int w = 1; w < 32; ++w) top = max(top, s_top[w]);
        *nlev = top;
    }
}

// The same on a cluster of CS blocks (512 threads each), for a level table
// in global memory: block c takes the steps c, c + CS, ... of every window
// (16 * CS / WR warps per step), so the scattered table reads and writes are
// spread over CS SMs. The steps' bases meet in distributed shared memory; a
// cluster barrier after the bases and one after the table writes keep the
// windows in order. *nlev must be zero at the start.
template <int WR, int CS>
__global__ void __launch_bounds__(512, 1) k_lvl_levels_cluster(
        const WinRow *__restrict__ rec, const unsigned char *__restrict__ dpath,
        const int32_t *__restrict__ oidx, int32_t nord, int32_t *lv, int32_t *__restrict__ lvl,
        int32_t *__restrict__ otag, int *__restrict__ nlev) {
    constexpr int RW = WR / CS;   // steps per block and window
    constexpr int WPR = 16 / RW;  // warps per step
    static_assert(CS == 16 && RW >= 2 && WPR >= 1 && RW * WPR == 16, "cluster shape");
    __shared__ int32_t base[RW], lvw[RW];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int rank = (int)cluster_rank();
    const int i = wid / WPR, sw = wid - i * WPR;  // the warp's step slot, warp in the step
    const WinRow none{0, 0, 0, 0, 0};
    const int nwin = (nord + WR - 1) / WR;
    int top = 0;
    // distributed shared memory address of the base of step `lane` of a window;
    // step lane + 32 j lies 2 j slots further in the same block
    uint32_t lane_base;
    {
        const uint32_t a = (uint32_t)__cvta_generic_to_shared(base);
        asm("mapa.shared::cluster.u32 %0, %1, %2;"
            : "=r"(lane_base)
            : "r"(a + 4u * (uint32_t)(lane / CS)), "r"((uint32_t)(lane % CS)));
    }
    const int r = rank + CS * i;  // this warp's step in every window
    WinRow wn = r < nord ? rec[r] : none;
    for (int q = 0; q < nwin; ++q) {
        const int k0 = q * WR, nr = min(WR, nord - k0);
        const bool mine = r < nr;
        const WinRow w = mine ? wn : none;
        if (sw == 0 && lane == 0) base[i] = 0;
        if (k0 + WR + r < nord) {  // the next window's step of this warp: its columns into L2
            wn = rec[k0 + WR + r];
            const char *c0 = reinterpret_cast<const char *>(oidx + wn.off);
            const int nl = (wn.len * 4 + 127) >> 7;
            for (int l = sw * 32 + lane; l < nl; l += 32 * WPR)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(c0 + ((size_t)l << 7)));
        }
        unsigned char d[WR / 32];
        if (mine && sw == 0)
#pragma unroll
            for (int j = 0; j < WR / 32; ++j) d[j] = dpath[(size_t)(k0 + r) * WR + 32 * j + lane];
        __syncthreads();
        if (mine) {  // 1 + the table's level over the step's first-touch columns
            int m = 0;
            for (int e0 = sw * 32 + lane; e0 < w.c2; e0 += 32 * WPR * 8) {
                int32_t j[8];
#pragma unroll
                for (int t = 0; t < 8; ++t) {
                    const int e = e0 + 32 * WPR * t;
                    j[t] = e < w.c2 ? oidx[w.off + e] : -1;
                }
#pragma unroll
                for (int t = 0; t < 8; ++t)
                    if (j[t] >= 0) {
                        const int32_t v = __ldcg(lv + j[t]);
                        m = max(m, v);
                        if (otag) otag[w.off + e0 + 32 * WPR * t] = v;
                    }
            }
            m = (int)__reduce_max_sync(0xffffffffu, (unsigned)m);
            if (lane == 0) atomicMax(&base[i], m + 1);
        }
        cluster_barrier();
        if (mine && sw == 0) {  // the longest paths within the window (of length d - 1)
            unsigned v = 0;
#pragma unroll
            for (int j = 0; j < WR / 32; ++j) {
                int bv = 0;
                if (d[j] > 0)
                    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(bv) : "r"(lane_base + 8u * j));
                if (d[j] > 0) v = max(v, (unsigned)(bv + d[j] - 1));
            }
            const int L = (int)__reduce_max_sync(0xffffffffu, v);
            if (lane == 0) {
                lvw[i] = L;
                lvl[k0 + r] = L;
            }
            top = max(top, L);
        }
        __syncthreads();
        if (mine) {  // the last touches of the window write the step's level
            const int L = lvw[i];
            for (int e0 = sw * 32 + lane; e0 < w.len; e0 += 32 * WPR * 8) {
                int32_t j[8];
#pragma unroll
                for (int t = 0; t < 8; ++t) {
                    const int e = e0 + 32 * WPR * t;
                    j[t] = e < w.len && (e < w.c1 || e >= w.c3) ? oidx[w.off + e] : -1;
                }
#pragma unroll
                for (int t = 0; t < 8; ++t)
                    if (j[t] >= 0) lv[j[t]] = L;
            }
        }
        cluster_barrier();
    }
    if (lane == 0 && top > 0) atomicMax(nlev, top);
}

// The same on a cooperative grid, a step of the window per block: the scattered
// table accesses are spread over up to WR SMs, and each thread's columns (the
// next window's loaded while a window runs) serve both phases from registers.
// The steps' bases are published as {window + 1, base} words that the blocks
// that need them poll (no barrier between the phases); a grid barrier closes the
// window. Fan N=512 (1901 windows of 128): 17.3 ms on the cluster, whose 16 SMs
// are bound by the scattered accesses (tags written), 8.5 ms here; N=128 1.11 and
// 0.79 ms.
template <int WR>
__global__ void __launch_bounds__(512, 1) k_lvl_levels_grid(
        const WinRow *__restrict__ rec, const unsigned char *__restrict__ dpath,
        const int32_t *__restrict__ oidx, int32_t nord, int32_t *lv, int32_t *__restrict__ lvl,
        int32_t *__restrict__ otag, unsigned long long *bases, unsigned *gbar, int *gerr,
        int *__restrict__ nlev) {
    constexpr int JC = 2, SW = WR / 32;  // columns per thread in registers; bases per lane
    __shared__ int s_max, s_level, s_ok;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int nwin = (nord + WR - 1) / WR;
    const int r = blockIdx.x;  // gridDim.x = WR: this block's step of every window
    const WinRow none{0, 0, 0, 0, 0};
    auto fetch = [&](const WinRow &w, int32_t (&j)[JC]) {
#pragma unroll
        for (int t = 0; t < JC; ++t) j[t] = tid + 512 * t < w.len ? __ldg(oidx + w.off + tid + 512 * t) : -1;
    };
    auto paths = [&](int k, unsigned char (&d)[SW]) {
#pragma unroll
        for (int i = 0; i < SW; ++i)
            d[i] = wid == 0 && k < nord ? __ldg(dpath + (size_t)k * WR + 32 * i + lane) : (unsigned char)0;
    };
    WinRow w = r < nord ? rec[r] : none, wn = WR + r < nord ? rec[WR + r] : none;
    int32_t j[JC];
    unsigned char d[SW];
    fetch(w, j);
    paths(r, d);
    if (tid == 0) {
        s_max = 0;
        s_ok = 1;
    }
    __syncthreads();
    int top = 0;
    for (int q = 0; q < nwin; ++q) {
        const int k = q * WR + r;
        const WinRow wn2 = k + 2 * WR < nord ? rec[k + 2 * WR] : none;
        int32_t jn[JC];
        unsigned char dn[SW];
        // 1 + the table's level over the step's first-touch columns
        int m = 0;
#pragma unroll
        for (int t = 0; t < JC; ++t) {
            const int e = tid + 512 * t;
            if (e < w.c2) {
                const int32_t v = __ldcg(lv + j[t]);
                m = max(m, v);
                if (otag) otag[w.off + e] = v;
            }
        }
        for (int e = tid + 512 * JC; e < w.c2; e += 512) {
            const int32_t v = __ldcg(lv + __ldg(oidx + w.off + e));
            m = max(m, v);
            if (otag) otag[w.off + e] = v;
        }
        fetch(wn, jn);
        paths(k + WR, dn);
        m = (int)__reduce_max_sync(0xffffffffu, (unsigned)m);
        if (lane == 0 && m > 0) atomicMax(&s_max, m);
        __syncthreads();
        unsigned long long *bq = bases + (q & 1) * WR;
        if (tid == 0 && k < nord) {
            const unsigned long long b = (unsigned long long)(unsigned)(q + 1) << 32 | (unsigned)(s_max + 1);
            asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(bq + r), "l"(b) : "memory");
        }
        if (wid == 0 && k < nord) {  // the longest paths within the window (of length d - 1)
            unsigned v = 0, need = 0;
#pragma unroll
            for (int i = 0; i < SW; ++i) need |= d[i] > 0 ? 1u << i : 0u;
            for (unsigned long long it = 1;; ++it) {
#pragma unroll
                for (int i = 0; i < SW; ++i)
                    if (need >> i & 1u) {
                        unsigned long long b;
                        asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(b) : "l"(bq + 32 * i + lane) : "memory");
                        if ((unsigned)(b >> 32) == (unsigned)(q + 1)) {
                            v = max(v, (unsigned)b + d[i] - 1u);
                            need &= ~(1u << i);
                        }
                    }
                if (__all_sync(0xffffffffu, need == 0)) break;
                if ((it & 1023u) == 0 && (it > kGridSpinLimit || *(volatile int *)gerr)) {
                    atomicExch(gerr, 1);
                    s_ok = 0;
                    break;
                }
            }
            const int L = (int)__reduce_max_sync(0xffffffffu, v);
            if (lane == 0) {
                s_level = L;
                s_max = 0;
                lvl[k] = L;
            }
            top = max(top, L);
        }
        __syncthreads();
        if (!s_ok) return;
        const int L = s_level;  // the last touches of the window write the step's level
#pragma unroll
        for (int t = 0; t < JC; ++t) {
            const int e = tid + 512 * t;
            if (e < w.len && (e < w.c1 || e >= w.c3)) lv[j[t]] = L;
        }
        for (int e = tid + 512 * JC; e < w.len; e += 512)
            if (e < w.c1 || e >= w.c3) lv[__ldg(oidx + w.off + e)] = L;
        if (!grid_barrier(gbar, gerr, (unsigned)q & 1u)) return;
        w = wn;
        wn = wn2;
#pragma unroll
        for (int t = 0; t < JC; ++t) j[t] = jn[t];
#pragma unroll
        for (int i = 0; i < SW; ++i) d[i] = dn[i];
    }
    if (tid == 0 && top > 0) atomicMax(nlev, top);
}

__global__ void k_lvl_count(const int32_t *__restrict__ lvl, int32_t nord, int32_t *cnt) {
    for (int32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < nord; k += gridDim.x * blockDim.x)
        atomicAdd(cnt + lvl[k] - 1, 1);
}
// steps in level order (any order within a level: its steps share no column),
// their levels beside them; eoff (when given): their first entries in the
// grouped arrays
__global__ void k_lvl_scatter(const RowStep *__restrict__ steps, const int32_t *__restrict__ lvl,
                              int32_t nord, const int64_t *__restrict__ lptr, int32_t *cnt,
                              const int64_t *__restrict__ eoff, RowStep *__restrict__ sched) {
    for (int32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < nord; k += gridDim.x * blockDim.x) {
        const int l = lvl[k] - 1;
        RowStep st = steps[k];
        st.level = l + 1;
        if (eoff) st.s = eoff[k];
        sched[lptr[l] + atomicSub(cnt + l, 1) - 1] = st;
    }
}
// Tags of the entries whose column an earlier step of their window has (a warp
// per step): that step's level.
template <int WR>
__global__ void k_lvl_tags(const WinRow *__restrict__ rec, int32_t nord, const int32_t *__restrict__ lvl,
                           int32_t *__restrict__ otag) {
    const int lane = threadIdx.x & 31;
    const int nw = (int)((gridDim.x * blockDim.x) >> 5);
    for (int k = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); k < nord; k += nw) {
        const WinRow w = rec[k];
        const int32_t *wl = lvl + k / WR * WR - 1;
        for (int e = w.c2 + lane; e < w.len; e += 32) otag[w.off + e] = wl[-otag[w.off + e]];
    }
}


// The schedule of the opposite direction: the levels and their steps in
// reverse (a step's level is above those of the earlier steps it shares a
// column with, so in reverse they come after it).
__global__ void k_lvl_reverse(const RowStep *__restrict__ sched, const int64_t *__restrict__ lptr,
                              const int *__restrict__ nlev, int32_t nord, RowStep *__restrict__ rsched,
                              int64_t *__restrict__ rlptr, int *__restrict__ rnlev) {
    const int L = *nlev;
    const int64_t t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, nt = (int64_t)gridDim.x * blockDim.x;
    for (int64_t k = t0; k < nord; k += nt) rsched[k] = sched[nord - 1 - k];
    for (int64_t l = t0; l <= L; l += nt) rlptr[l] = nord - lptr[L - l];
    if (t0 == 0) *rnlev = L;
}

// Where the level sweep keeps x: global memory read past L1 (XG), the
// block's shared memory (XS, one block), or the cluster's distributed shared
// memory (XD: block r holds x[r * 2^cb, (r + 1) * 2^cb)). XS and XD address x
// by 32-bit shared-window addresses.
enum { XG = 0, XS = 1, XD = 2 };
template <int XM> struct XAcc;
template <> struct XAcc<XG> {
    double *x;
    using R = double *;
    __device__ __forceinline__ R ref(int32_t j) const { return x + j; }
    __device__ __forceinline__ double ld(R p) const { return __ldcg(p); }
    __device__ __forceinline__ void st(R p, double v) const { *p = v; }
};
template <> struct XAcc<XS> {
    uint32_t base;  // shared-window address of x
    using R = uint32_t;
    __device__ __forceinline__ R ref(int32_t j) const { return base + ((uint32_t)j << 3); }
    __device__ __forceinline__ double ld(R a) const {
        double v;
        asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a));
        return v;
    }
    __device__ __forceinline__ void st(R a, double v) const {
        asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v));
    }
};
template <> struct XAcc<XD> {
    uint32_t base;  // shared-window address of this block's part
    int cb;         // log2 of the part's length
    using R = uint32_t;
    __device__ __forceinline__ R ref(int32_t j) const {  // an address, no memory access
        const uint32_t a = base + (((uint32_t)j & ((1u << cb) - 1u)) << 3);
        uint32_t r;
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"((uint32_t)j >> cb));
        return r;
    }
    // volatile keeps these in program order among themselves and against the
    // barriers (also volatile asm), the only ordering the sweep needs
    __device__ __forceinline__ double ld(R a) const {
        double v;
        asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a));
        return v;
    }
    __device__ __forceinline__ void st(R a, double v) const {
        asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v));
    }
};

// A warp's first CACHE chunks of a step (column and value of entry lane of
// each chunk; column 0 and value 0 past the row's end).
template <int CACHE> struct LvlChunks {
    int32_t c[CACHE];
    double v[CACHE];
};
template <int CACHE>
__device__ __forceinline__ void lvl_load_chunks(const RowStep &st, const int32_t *__restrict__ col,
                                                const double *__restrict__ val, int lane, int G,
                                                int wg, LvlChunks<CACHE> &k) {
    const int nq = (st.len + 31) >> 5;
    const int nmine = nq > wg ? (nq - wg + G - 1) / G : 0;
#pragma unroll
    for (int i = 0; i < CACHE; ++i) {
        const int e = (wg + G * i) * 32 + lane;
        const bool h = i < nmine && e < st.len;
        k.c[i] = h ? __ldg(col + st.s + e) : 0;
        k.v[i] = h ? __ldg(val + st.s + e) : 0.0;
    }
}

// The coefficient -(a.x - b) (omega / nrA) of a group's step from its warps'
// parts (of shared memory: parts, G each, and coef). WIDE: G may be 16 (fx_group's
// test lies on every level's chain: fan N=128 without barriers, G = 8, 19.91 ms with
// it and 19.79 without).
template <bool WIDE>
__device__ __forceinline__ double step_coef(const FxPart &part, FxPart *parts, double *coef, int G, int wg,
                                            int lane, int bar, double w) {
    if (G > 1) {
        // by one warp of the group for all: the G parts one per lane, aligned and
        // added by warp reductions. All 16 warps of a block at it (the conversion
        // and the product are 64 cycles each of a sub-partition's FP64 pipe, and
        // about 200 integer instructions where they are done without it) took 730
        // of a level's 5650 cycles at fan N=128 and 1410 of 8800 at N=512 (sweeps
        // 3.22 and 13.2 ms; one warp: 2.72 and 12.6 ms); groups take warps of
        // different sub-partitions.
        if (lane == 0) parts[wg] = part;
        asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(32 * G) : "memory");
        if (wg == (bar & (G - 1))) {
            const int e = lane < G ? parts[lane].e : 0;
            const int E = (int)__reduce_max_sync(0xffffffffu, (unsigned)e);
            double r;
            if (E >= 0x7FF) {
                r = fx_special(parts, G);
            } else {
                const int sh = E - e;
                const long long F = lane < G && sh < 64 ? parts[lane].s >> sh : 0ll;
                r = WIDE ? fx_group(F, E) : fx_to_double_fast(fx_warp_sum(F), E);
            }
            if (lane == 0) *coef = __dmul_rn(-r, w);
        }
        asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(32 * G) : "memory");
        return *(volatile double *)coef;
    }
    return __dmul_rn(-(part.e >= 0x7FF ? part.d : fx_to_double_fast(part.s, part.e)), w);
}

// One step by a group of G warps: the row's chunks of 32 entries are dealt
// to the group's warps in turn (chunk q to warp q mod G), CACHE chunks per
// warp held in registers and the rest loaded in batches of four. Each warp's
// part of a.x - b is an exact fixed-point sum (fx_warp_part); the G parts meet
// in shared memory behind the group's named barrier, are added exactly and
// rounded once; then the coefficient (b - a.x) * (omega / nrA) and the bounded
// updates.
template <int XM, int CACHE>
__device__ __forceinline__ void lvl_row(const RowStep &st, const int32_t *__restrict__ col,
                                        const double *__restrict__ val, const XAcc<XM> &X,
                                        const Box &box, int lane, int G, int wg, FxPart *parts,
                                        double *coef, int bar, const LvlChunks<CACHE> &pre) {
    using R = typename XAcc<XM>::R;
    constexpr int B = 4;  // chunks per batch beyond the cached ones
    R cr[CACHE];
    double vv[CACHE], xo[CACHE];
    const int nq = (st.len + 31) >> 5;                      // chunks of the row
    const int nmine = nq > wg ? (nq - wg + G - 1) / G : 0;  // this warp's chunks
    int32_t cj[CACHE];
#pragma unroll
    for (int i = 0; i < CACHE; ++i) {
        cj[i] = pre.c[i];
        vv[i] = pre.v[i];
    }
#pragma unroll
    for (int i = 0; i < CACHE; ++i) {
        if (i >= nmine) break;
        cr[i] = X.ref(cj[i]);
    }
#pragma unroll
    for (int i = 0; i < CACHE; ++i) {
        if (i >= nmine) break;
        xo[i] = (wg + G * i) * 32 + lane < st.len ? X.ld(cr[i]) : 0.0;
    }
    double p0 = 0.0, p1 = 0.0;
#pragma unroll
    for (int i = 0; i < CACHE; ++i) {
        if (i >= nmine) break;
        if (i & 1) p1 = fma(xo[i], vv[i], p1);
        else p0 = fma(xo[i], vv[i], p0);
    }
    for (int i0 = CACHE; i0 < nmine; i0 += B) {
        R tr[B];
        bool th[B];
        double tv[B], tx[B];
        int32_t tj[B];
#pragma unroll
        for (int t = 0; t < B; ++t) {
            const int e = (wg + G * (i0 + t)) * 32 + lane;
            th[t] = i0 + t < nmine && e < st.len;
            tj[t] = th[t] ? __ldg(col + st.s + e) : 0;
            tv[t] = th[t] ? __ldg(val + st.s + e) : 0.0;
        }
#pragma unroll
        for (int t = 0; t < B; ++t) tr[t] = X.ref(tj[t]);
#pragma unroll
        for (int t = 0; t < B; ++t) tx[t] = th[t] ? X.ld(tr[t]) : 0.0;
#pragma unroll
        for (int t = 0; t < B; ++t) {
            if (t & 1) p1 = fma(tx[t], tv[t], p1);
            else p0 = fma(tx[t], tv[t], p0);
        }
    }
    const FxPart part = fx_warp_part(p0, p1, (wg == 0 && lane == 0) ? -st.b : 0.0);
    const double c = step_coef<true>(part, parts, coef, G, wg, lane, bar, st.w);
#pragma unroll
    for (int i = 0; i < CACHE; ++i) {
        if (i >= nmine) break;
        if ((wg + G * i) * 32 + lane < st.len) X.st(cr[i], box.apply(fma(c, vv[i], xo[i])));
    }
    for (int i0 = CACHE; i0 < nmine; i0 += B) {
        R tr[B];
        bool th[B];
        double tv[B], tx[B];
        int32_t tj[B];
#pragma unroll
        for (int t = 0; t < B; ++t) {
            const int e = (wg + G * (i0 + t)) * 32 + lane;
            th[t] = i0 + t < nmine && e < st.len;
            tj[t] = th[t] ? __ldg(col + st.s + e) : 0;
            tv[t] = th[t] ? __ldg(val + st.s + e) : 0.0;
        }
#pragma unroll
        for (int t = 0; t < B; ++t) tr[t] = X.ref(tj[t]);
#pragma unroll
        for (int t = 0; t < B; ++t) tx[t] = th[t] ? X.ld(tr[t]) : 0.0;
#pragma unroll
        for (int t = 0; t < B; ++t)
            if (th[t]) X.st(tr[t], box.apply(fma(c, tv[t], tx[t])));
    }
}


enum { SYNC_BLOCK = 0, SYNC_CLUSTER = 1, SYNC_GRID = 2 };

// The levels in order on one cluster of gridDim.x blocks (CLUSTER) or one
// block. Groups of G consecutive warps take the steps of a level in turn; each
// group's first step of a level is known two levels ahead and its first
// chunks are loaded one level ahead (in registers). With x in
// (distributed) shared memory (XM = XS or XD, cb = log2 of a block's part), x
// is loaded at the start and written back at the end.
template <int SYNC, int XM, int CACHE, int NT>
__global__ void __launch_bounds__(NT, 1) k_lvl_sweep(
        const RowStep *__restrict__ sched, const int64_t *__restrict__ lptr,
        const int *__restrict__ nlevp, const int32_t *__restrict__ col,
        const double *__restrict__ val, double *x, int32_t n, int cb, Box box, int G,
        const int *__restrict__ err, unsigned *gbar, int *gerr) {
    constexpr int NW = NT / 32;
    constexpr bool CLUSTER = SYNC == SYNC_CLUSTER;
    extern __shared__ __align__(16) double xsm[];
    __shared__ FxPart parts[2][NW];  // per group: two rows' parts (by parity), G each
    __shared__ double coef[2][NW];
    if (*err) return;
    const int nlev = *nlevp;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    XAcc<XM> X;
    int64_t part0 = 0, plen = 0;  // this block's part of x (XS: all of it)
    if constexpr (XM == XG) {
        X.x = x;
    } else {
        X.base = (uint32_t)__cvta_generic_to_shared(xsm);
        if constexpr (XM == XD) {
            X.cb = cb;
            part0 = (int64_t)cluster_rank() << cb;
            plen = (int64_t)1 << cb;
        } else {
            plen = n;
        }
        for (int64_t i = threadIdx.x; i < plen; i += NT)
            xsm[i] = part0 + i < n ? x[part0 + i] : 0.0;
    }
    if (CLUSTER) cluster_barrier();
    else __syncthreads();
    const int gl = wid / G, wg = wid - gl * G;  // group in the block, warp in the group
    const int64_t grp = (int64_t)blockIdx.x * (NW / G) + gl;
    const int64_t NG = (int64_t)gridDim.x * (NW / G);
    const int bar = 1 + gl;
    const RowStep none{0, 0, 0, 0.0, 0.0};
    // State at the start of level l: the bounds of levels l, l+1, l+2
    // ([a0, a1), [a1, a2), [a2, a3)); this group's first step of level l (cur,
    // its first chunks in pc) and of level l+1 (nxt). During level l the group
    // loads the bound after a3, its first step of level l+2 and the first
    // chunks of nxt, so that no level waits for a load of its own bounds,
    // steps or first entries; the rest of nxt's entries are prefetched into L2.
    auto bound = [&](int q) -> int64_t { return q <= nlev ? lptr[q] : lptr[nlev]; };
    int64_t a0 = 0, a1 = bound(1), a2 = bound(2), a3 = bound(3);
    RowStep cur = grp < a1 ? sched[grp] : none;
    RowStep nxt = a1 + grp < a2 ? sched[a1 + grp] : none;
    LvlChunks<CACHE> pc;
    lvl_load_chunks<CACHE>(cur, col, val, lane, G, wg, pc);
    for (int l = 0; l < nlev; ++l) {
        const int64_t a4 = bound(l + 4);
        const RowStep nxt2 = a2 + grp < a3 ? sched[a2 + grp] : none;
        LvlChunks<CACHE> pn;
        lvl_load_chunks<CACHE>(nxt, col, val, lane, G, wg, pn);
        int par = 0;
        for (int64_t k = a0 + grp; k < a1; k += NG, par ^= 1) {
            if (k == a0 + grp) {
                lvl_row<XM, CACHE>(cur, col, val, X, box, lane, G, wg, parts[par] + gl * G, &coef[par][gl], bar, pc);
            } else {
                const RowStep st = sched[k];
                LvlChunks<CACHE> pk;
                lvl_load_chunks<CACHE>(st, col, val, lane, G, wg, pk);
                lvl_row<XM, CACHE>(st, col, val, X, box, lane, G, wg, parts[par] + gl * G, &coef[par][gl], bar, pk);
            }
        }
        if (nxt.len > 32 * G * CACHE) {  // the rest of the next level's first step: into L2
            const char *c0 = reinterpret_cast<const char *>(col + nxt.s);
            const char *v0 = reinterpret_cast<const char *>(val + nxt.s);
            const int nc = (nxt.len * 4 + 127) >> 7, nv = (nxt.len * 8 + 127) >> 7;
            for (int i = wg * 32 + lane; i < nc + nv; i += 32 * G) {
                const char *p = i < nc ? c0 + ((size_t)i << 7) : v0 + ((size_t)(i - nc) << 7);
                asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
            }
        }
        if (SYNC == SYNC_CLUSTER) cluster_barrier();
        else if (SYNC == SYNC_GRID) {
            if (!grid_barrier(gbar, gerr, (unsigned)l & 1u)) return;
        } else {
            __syncthreads();
        }
        a0 = a1;
        a1 = a2;
        a2 = a3;
        a3 = a4;
        cur = nxt;
        nxt = nxt2;
        pc = pn;
    }
    if constexpr (XM != XG) {
        for (int64_t i = threadIdx.x; i < plen; i += NT)
            if (part0 + i < n) x[part0 + i] = xsm[i];
    }
}

// ---- the sweep without barriers -------------------------------------------------
// Between two levels of a barrier sweep lie a release of the writes, a barrier
// and the reads of x, each a round trip through L2, and every step waits for
// the slowest of its level. Here each x_j is kept as a 16-byte pair {value,
// level of the last step that updated it}, read and written whole (128-bit
// relaxed accesses are single-copy atomic), and each entry carries the level
// its column must have reached (its tag: the level of the column's last
// earlier step, from the level set-up). A group of G warps takes the steps grp,
// grp + groups, ... of the level schedule, polls its entries' pairs until
// each shows its tag, and writes them back with the step's own level: the
// value is its own signal, so a step starts as soon as its last column
// arrives, one store and one load after its predecessor. Every toucher of a
// column updates it, so no version is missed or overwritten before its one
// reader has seen it.
// The blocks are co-resident (a cooperative launch) and every group takes its
// steps in schedule order, so the first unfinished step of the schedule always
// finds its columns ready. A wait longer than kGridSpinLimit polls sets *gerr;
// all waits then end (checked every 1024 polls), and the host reports the error.
// Bound by the latency of one level's chain: a store and a poll through L2, the
// row's FP64 products, the parts' exchange. Per sweep, fan N=128 (1019 levels)
// 2.72 ms on the cluster with x in distributed shared memory, 1.79 ms here; N=512
// (3018 levels) 12.6 ms on the grid with barriers, 9.1 ms here.
struct __align__(16) XPair {
    double v;
    long long level;
};
__device__ __forceinline__ void pair_ld(const XPair *p, double &v, long long &level) {
    long long b;
    asm volatile("{\n.reg .b128 t;\nld.relaxed.gpu.global.b128 t, [%2];\nmov.b128 {%0, %1}, t;\n}"
                 : "=l"(b), "=l"(level) : "l"(p) : "memory");
    v = __longlong_as_double(b);
}
__device__ __forceinline__ void pair_st(XPair *p, double v, long long level) {
    asm volatile("{\n.reg .b128 t;\nmov.b128 t, {%1, %2};\nst.relaxed.gpu.global.b128 [%0], t;\n}"
                 ::"l"(p), "l"(__double_as_longlong(v)), "l"(level) : "memory");
}
__global__ void k_flow_pack(const double *__restrict__ x, int32_t n, XPair *__restrict__ xt) {
    for (int32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x)
        xt[j] = XPair{x[j], 0};
}
__global__ void k_flow_unpack(const XPair *__restrict__ xt, int32_t n, double *__restrict__ x) {
    for (int32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) x[j] = xt[j].v;
}

template <int K> struct FlowChunks {  // entries of a warp's chunks: column (-1: none), value, tag
    int32_t c[K], t[K];
    double v[K];
};
template <int K>
__device__ __forceinline__ void flow_load(const RowStep &st, const int32_t *__restrict__ col,
                                          const double *__restrict__ val, const int32_t *__restrict__ tag,
                                          int lane, int G, int q0, FlowChunks<K> &k) {
#pragma unroll
    for (int i = 0; i < K; ++i) {
        const int e = (q0 + G * i) * 32 + lane;
        const bool h = e < st.len;
        k.c[i] = h ? __ldg(col + st.s + e) : -1;
        k.t[i] = h ? __ldg(tag + st.s + e) : 0;
        k.v[i] = h ? __ldg(val + st.s + e) : 0.0;
    }
}
// The values of the chunks' columns, each once it has its tag (dead: a wait has
// run out, no more waiting).
template <int K>
__device__ __forceinline__ void flow_wait(const FlowChunks<K> &k, const XPair *xt, double (&xo)[K], bool &dead,
                                          int *gerr) {
    unsigned need = 0;
#pragma unroll
    for (int i = 0; i < K; ++i) {
        xo[i] = 0.0;
        if (k.c[i] >= 0) need |= 1u << i;
    }
    for (unsigned long long it = 1;; ++it) {
        double v[K];
        long long l[K];
#pragma unroll
        for (int i = 0; i < K; ++i)
            if (need >> i & 1u) pair_ld(xt + k.c[i], v[i], l[i]);
#pragma unroll
        for (int i = 0; i < K; ++i)
            if ((need >> i & 1u) && l[i] == (long long)k.t[i]) {
                xo[i] = v[i];
                need &= ~(1u << i);
            }
        if (__all_sync(0xffffffffu, need == 0) || dead) break;
        if ((it & 1023u) == 0 && (it > kGridSpinLimit || *(volatile int *)gerr)) {
            dead = true;
            atomicExch(gerr, 1);
        }
    }
}

template <int CACHE, int NT, bool WIDE>
__global__ void __launch_bounds__(NT, 1) k_flow_sweep(
        const RowStep *__restrict__ sched, int32_t nord, const int32_t *__restrict__ col,
        const double *__restrict__ val, const int32_t *__restrict__ tag, XPair *xt, Box box, int G,
        const int *__restrict__ err, int *gerr) {
    constexpr int NW = NT / 32, B = 2;  // B: chunks per batch beyond the cached ones
    __shared__ FxPart parts[2][NW];
    __shared__ double coef[2][NW];
    if (*err) return;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int gl = wid / G, wg = wid - gl * G, bar = 1 + gl;
    // consecutive steps on different SMs
    const int64_t grp = (int64_t)gl * gridDim.x + blockIdx.x, NG = (int64_t)gridDim.x * (NW / G);
    const RowStep none{0, 0, 0, 0.0, 0.0};
    bool dead = false;
    RowStep cur = grp < nord ? sched[grp] : none, nxt = grp + NG < nord ? sched[grp + NG] : none;
    FlowChunks<CACHE> pc;
    flow_load<CACHE>(cur, col, val, tag, lane, G, wg, pc);
    int par = 0;
    for (int64_t k = grp; k < nord; k += NG, par ^= 1) {
        const RowStep nxt2 = k + 2 * NG < nord ? sched[k + 2 * NG] : none;
        FlowChunks<CACHE> pn;
        flow_load<CACHE>(nxt, col, val, tag, lane, G, wg, pn);
        const int nq = (cur.len + 31) >> 5;
        double xo[CACHE];
        flow_wait<CACHE>(pc, xt, xo, dead, gerr);
        double p0 = 0.0, p1 = 0.0;
#pragma unroll
        for (int i = 0; i < CACHE; ++i) {
            if (wg + G * i >= nq) break;
            if (i & 1) p1 = fma(xo[i], pc.v[i], p1);
            else p0 = fma(xo[i], pc.v[i], p0);
        }
        for (int q0 = wg + G * CACHE; q0 < nq; q0 += G * B) {
            FlowChunks<B> f;
            double x2[B];
            flow_load<B>(cur, col, val, tag, lane, G, q0, f);
            flow_wait<B>(f, xt, x2, dead, gerr);
            p0 = fma(x2[0], f.v[0], p0);
            p1 = fma(x2[1], f.v[1], p1);
        }
        const FxPart part = fx_warp_part(p0, p1, (wg == 0 && lane == 0) ? -cur.b : 0.0);
        const double c = step_coef<WIDE>(part, parts[par] + gl * G, &coef[par][gl], G, wg, lane, bar, cur.w);
#pragma unroll
        for (int i = 0; i < CACHE; ++i) {
            if (wg + G * i >= nq) break;
            if (pc.c[i] >= 0) pair_st(xt + pc.c[i], box.apply(fma(c, pc.v[i], xo[i])), cur.level);
        }
        for (int q0 = wg + G * CACHE; q0 < nq; q0 += G * B) {
            FlowChunks<B> f;
            flow_load<B>(cur, col, val, tag, lane, G, q0, f);
#pragma unroll
            for (int i = 0; i < B; ++i)
                if (f.c[i] >= 0) {  // this step's until it writes it
                    double v;
                    long long l;
                    pair_ld(xt + f.c[i], v, l);
                    pair_st(xt + f.c[i], box.apply(fma(c, f.v[i], v)), cur.level);
                }
        }
        cur = nxt;
        nxt = nxt2;
        pc = pn;
    }
}

int env_int(const char *name, int dflt) {
    const char *v = getenv(name);
    return v && *v ? atoi(v) : dflt;
}

// log2 of the power-of-two part of x per block when cs blocks hold n entries
int part_log2(int cs, int32_t n) {
    int cb = 0;
    while (((int64_t)cs << cb) < (int64_t)n) ++cb;
    return cb;
}

// The cluster shape of the level sweep: the largest of 16, 8, 4, 2 blocks
// (at most `want`) that the device can co-schedule, each with its part of x
// in shared memory (XD: 8 << part_log2 bytes, at most `room`) or none (XG);
// 1 if none can be had.
template <int XM, int CACHE, int NT>
int lvl_cluster_size(int want, int32_t n, size_t room) {
    auto kern = k_lvl_sweep<SYNC_CLUSTER, XM, CACHE, NT>;
    for (int cs = 16; cs >= 2; cs >>= 1) {
        if (cs > want) continue;
        const size_t smem = XM == XD ? (size_t)8 << part_log2(cs, n) : 0;
        if (XM == XD && smem > room) continue;
        if (smem_allow(reinterpret_cast<const void *>(kern), smem) != cudaSuccess ||
            (cs > 8 && cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)) {
            cudaGetLastError();
            continue;
        }
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(cs);
        cfg.blockDim = dim3(NT);
        cfg.dynamicSmemBytes = smem;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = cs;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int nc = 0;
        if (cudaOccupancyMaxActiveClusters(&nc, kern, &cfg) == cudaSuccess && nc >= 1) return cs;
        cudaGetLastError();
    }
    return 1;
}

template <int XM, int CACHE, int NT>
int lvl_launch_cluster(int cs, size_t smem, const RowStep *sched, const int64_t *lptr,
                       const int *nlev, const int32_t *col, const double *val, double *x,
                       int32_t n, int cb, const Box &box, int G, const int *err, cudaStream_t s) {
    auto kern = k_lvl_sweep<SYNC_CLUSTER, XM, CACHE, NT>;
    FAIR_CUDA(smem_allow(reinterpret_cast<const void *>(kern), smem));
    if (cs > 8) FAIR_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(cs);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cs;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    FAIR_CUDA(cudaLaunchKernelEx(&cfg, kern, sched, lptr, nlev, col, val, x, n, cb, box, G, err,
                                 (unsigned *)nullptr, (int *)nullptr));
    return FAIR_OK;
}

// Launches the level sweep: x in the distributed shared memory of a cluster
// when its parts (a power of two per block) fit, else in global memory; one
// block with x in its shared memory when no cluster can be had.
// FAIR_SWEEP_CLUSTER caps the cluster size (1: one block), FAIR_SWEEP_XMEM
// picks x's place (0: global, 1: shared/distributed).
// The level sweep on a cooperative grid of nb blocks (x in global memory, the
// software grid barrier between levels); gsync: {barrier counter, unused, error}.
// *ran = false where the cooperative launch is refused.
template <int CACHE, int NT>
int lvl_launch_grid(int nb, const RowStep *sched, const int64_t *lptr, const int *nlev,
                    const int32_t *col, const double *val, double *x, int32_t n, const Box &box,
                    int G, const int *err, int *gsync, cudaStream_t s, bool *ran) {
    auto kern = k_lvl_sweep<SYNC_GRID, XG, CACHE, NT>;
    FAIR_CUDA(cudaMemsetAsync(gsync, 0, 4 * sizeof(int), s));
    *ran = launch_cooperative(nb, NT, s, kern, sched, lptr, nlev, col, val, x, n, 0, box, G, err,
                              (unsigned *)gsync, gsync + 2);
    if (!*ran) return FAIR_OK;
    int gerr = 0;
    FAIR_CUDA(cudaMemcpyAsync(&gerr, gsync + 2, sizeof(int), cudaMemcpyDeviceToHost, s));
    FAIR_CUDA(cudaStreamSynchronize(s));
    if (gerr) {
        set_detail("Kaczmarz level sweep: a grid barrier timed out");
        return FAIR_ERR_CUDA;
    }
    return FAIR_OK;
}

// Blocks of a cooperative grid for a level sweep whose levels hold `spl`
// steps of G warps on average (room for twice that: the wavefront's levels
// vary), at most the co-resident blocks; 0 when the grid would not exceed the
// cluster (cs blocks).
template <int CACHE, int NT>
int lvl_grid_blocks(double spl, int G, int cs) {
    int want = (int)std::ceil(spl * 2.0 * G / (NT / 32));
    // FAIR_SWEEP_GRID_BLOCKS sets the count instead (tuning measurements),
    // still capped at the co-resident blocks
    const int forced = env_int("FAIR_SWEEP_GRID_BLOCKS", 0);
    if (forced > 0) want = forced;
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_lvl_sweep<SYNC_GRID, XG, CACHE, NT>, NT, 0) !=
            cudaSuccess || occ < 1) {
        cudaGetLastError();
        return 0;
    }
    const int nb = std::min(want, occ * sm_count());
    return nb > cs ? nb : 0;
}

template <int CACHE, int NT>
int lvl_launch(const SweepDev &S, const RowStep *sched, const int64_t *lptr, const int *nlev,
               const int32_t *col, const double *val, const Box &box, int G, const int *err, double spl,
               cudaStream_t s) {
    // cluster sizes found per device, x placement and image size (host
    // threads may sweep on different handles at once)
    static struct { int32_t n = -1; int want = 0, cs = 0; } cache[128][2];
    static std::mutex cache_mu;
    int dev = 0, optin = 0;
    FAIR_CUDA(cudaGetDevice(&dev));
    FAIR_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    const int want = std::max(1, env_int("FAIR_SWEEP_CLUSTER", 16));
    const bool xmem = env_int("FAIR_SWEEP_XMEM", 1) != 0;
    const int32_t n = S.A->n;
    const size_t room = (size_t)optin - 8192;  // beside the static parts
    auto cluster = [&](int xd) {
        std::lock_guard<std::mutex> lk(cache_mu);
        auto &c = cache[dev & 127][xd];
        if (c.n != n || c.want != want) {
            c.cs = xd ? lvl_cluster_size<XD, CACHE, NT>(want, n, room)
                      : lvl_cluster_size<XG, CACHE, NT>(want, n, room);
            c.n = n;
            c.want = want;
        }
        return c.cs;
    };
    // levels with more steps than one round of the cluster's groups: a
    // cooperative grid (FAIR_SWEEP_GRID=0 keeps the cluster, 1 forces the grid)
    {
        const int gmode = env_int("FAIR_SWEEP_GRID", -1);
        const int cs = cluster(xmem ? 1 : 0);
        int nb = gmode == 0 ? 0 : lvl_grid_blocks<CACHE, NT>(spl, G, std::max(cs, 1));
        if (gmode == 1 && nb == 0) nb = std::min(2 * std::max(cs, 1), sm_count());
        bool ran = false;
        if (nb > 0 && S.work)
            FAIR_TRY((lvl_launch_grid<CACHE, NT>(nb, sched, lptr, nlev, col, val, S.x, n, box, G, err,
                                                 S.work->gsync.as<int>(), s, &ran)));
        if (ran) return FAIR_OK;
    }
    if (xmem) {
        const int cs = cluster(1);
        if (cs >= 2) {
            const int cb = part_log2(cs, n);
            return lvl_launch_cluster<XD, CACHE, NT>(cs, (size_t)8 << cb, sched, lptr, nlev, col, val,
                                                     S.x, n, cb, box, G, err, s);
        }
        if ((size_t)8 * n <= room) {
            auto kern = k_lvl_sweep<SYNC_BLOCK, XS, CACHE, NT>;
            FAIR_CUDA(smem_allow(reinterpret_cast<const void *>(kern), 8 * (size_t)n));
            kern<<<1, NT, 8 * (size_t)n, s>>>(sched, lptr, nlev, col, val, S.x, n, 0, box, G, err, nullptr,
                                               nullptr);
            FAIR_CUDA(cudaGetLastError());
            return FAIR_OK;
        }
    }
    const int cs = cluster(0);
    if (cs <= 1) {
        k_lvl_sweep<SYNC_BLOCK, XG, CACHE, NT><<<1, NT, 0, s>>>(sched, lptr, nlev, col, val, S.x, n,
                                                               0, box, G, err, nullptr, nullptr);
        FAIR_CUDA(cudaGetLastError());
        return FAIR_OK;
    }
    return lvl_launch_cluster<XG, CACHE, NT>(cs, 0, sched, lptr, nlev, col, val, S.x, n, 0, box, G,
                                             err, s);
}

// The sweep without barriers on a cooperative grid of nb blocks (*ran = false, x as
// it was, where that launch is refused); gsync: {unused, unused, error}.
template <int CACHE, int NT, bool WIDE>
int flow_launch(int nb, const RowStep *sched, int32_t nord, const int32_t *col, const double *val,
                const int32_t *tag, XPair *xt, double *x, int32_t n, const Box &box, int G, const int *err,
                int *gsync, cudaStream_t s, bool *ran) {
    auto kern = k_flow_sweep<CACHE, NT, WIDE>;
    FAIR_CUDA(cudaMemsetAsync(gsync, 0, 4 * sizeof(int), s));
    const int g = (int)std::max<int64_t>(1, std::min<int64_t>(((int64_t)n + 255) / 256, (int64_t)sm_count() * 8));
    k_flow_pack<<<g, 256, 0, s>>>(x, n, xt);
    *ran = launch_cooperative(nb, NT, s, kern, sched, nord, col, val, tag, xt, box, G, err, gsync + 2);
    if (!*ran) return FAIR_OK;
    k_flow_unpack<<<g, 256, 0, s>>>(xt, n, x);
    FAIR_CUDA(cudaGetLastError());
    int gerr = 0;
    FAIR_CUDA(cudaMemcpyAsync(&gerr, gsync + 2, sizeof(int), cudaMemcpyDeviceToHost, s));
    FAIR_CUDA(cudaStreamSynchronize(s));
    if (gerr) {
        set_detail("Kaczmarz sweep: a step waited too long for its columns");
        return FAIR_ERR_CUDA;
    }
    return FAIR_OK;
}

// The levels on a 16-block cluster (the level table in global memory);
// false when no such cluster can be had (FAIR_SWEEP_CLUSTER below 16 also
// keeps the single block).
template <int WR>
bool lvl_levels_cluster(SweepWork &W, int32_t nord, int *nlev, int32_t *otag, cudaStream_t s) {
    if (env_int("FAIR_SWEEP_CLUSTER", 16) < 16) return false;
    auto kern = k_lvl_levels_cluster<WR, 16>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(16);
    cfg.blockDim = dim3(512);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 16;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int nc = 0;
    if (cudaOccupancyMaxActiveClusters(&nc, kern, &cfg) != cudaSuccess || nc < 1) {
        cudaGetLastError();
        return false;
    }
    if (cudaMemsetAsync(nlev, 0, sizeof(int), s) != cudaSuccess ||
        cudaLaunchKernelEx(&cfg, kern, (const WinRow *)W.rec.as<WinRow>(),
                           (const unsigned char *)W.dpath.as<unsigned char>(),
                           (const int32_t *)W.idx.as<int32_t>(), nord, W.lvtab.as<int32_t>(),
                           W.lvl.as<int32_t>(), otag, nlev) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return true;
}

// The levels on a cooperative grid of WR blocks (a step of every window each);
// false when the device cannot hold them at once (FAIR_SWEEP_CLUSTER also keeps
// to the cluster). gsync: {barrier counter, -, error}, read by the caller.
template <int WR>
bool lvl_levels_grid(SweepWork &W, int32_t nord, int *nlev, int32_t *otag, cudaStream_t s) {
    if (getenv("FAIR_SWEEP_CLUSTER")) return false;
    auto kern = k_lvl_levels_grid<WR>;
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, 512, 0) != cudaSuccess || occ * sm_count() < WR ||
        W.bases.grow(2 * WR * sizeof(unsigned long long))) {
        cudaGetLastError();
        return false;
    }
    if (cudaMemsetAsync(nlev, 0, sizeof(int), s) != cudaSuccess ||
        cudaMemsetAsync(W.bases.p, 0, 2 * WR * sizeof(unsigned long long), s) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return launch_cooperative(WR, 512, s, kern, (const WinRow *)W.rec.as<WinRow>(),
                              (const unsigned char *)W.dpath.as<unsigned char>(),
                              (const int32_t *)W.idx.as<int32_t>(), nord, W.lvtab.as<int32_t>(),
                              W.lvl.as<int32_t>(), otag, W.bases.as<unsigned long long>(), W.gsync.as<unsigned>(),
                              W.gsync.as<int>() + 2, nlev);
}

// Set-up and levels in windows of WR steps. *built = false (and FAIR_OK) when
// a buffer cannot be had.
template <int WR>
int lvl_build(const SweepDev &S, SweepWork &W, SweepWork::Levels &C, const RowStep *steps, size_t setup_smem,
              size_t optin, bool want, bool flow, bool *built, cudaStream_t s) {
    const DevCSR &A = *S.A;
    const int32_t nord = S.nord;
    const int nwin = (nord + WR - 1) / WR;
    const size_t tab_row = (size_t)std::max<int32_t>(A.n, 1) * sizeof(unsigned long long);
    int blocks = std::min(nwin, 2 * sm_count());
    blocks = (int)std::max<size_t>(1, std::min<size_t>((size_t)blocks, ((size_t)2 << 30) / tab_row));
    int32_t *otag = flow ? W.tag.as<int32_t>() : nullptr;
    *built = false;
    if (W.dpath.grow((size_t)WR * ((size_t)nord + WR))) return FAIR_OK;
    if (W.tab_n != A.n || W.tab_blocks < blocks || W.uid + (uint64_t)nwin >= kStampIdLimit) {
        W.tabs.release();
        W.tab_n = 0;
        W.tab_blocks = 0;
        if (W.tabs.grow(tab_row * (size_t)blocks)) return FAIR_OK;
        FAIR_CUDA(cudaMemsetAsync(W.tabs.p, 0xFF, tab_row * (size_t)blocks, s));
        W.tab_n = A.n;
        W.tab_blocks = blocks;
        W.uid = 0;
    }
    FAIR_CUDA(smem_allow(reinterpret_cast<const void *>(k_lvl_setup<WR>), setup_smem));
    k_lvl_setup<WR><<<blocks, kSetupThreads, setup_smem, s>>>(
        steps, W.eoff.as<int64_t>(), nord, A.col.as<int32_t>(), W.tabs.as<unsigned long long>(), A.n, W.uid,
        W.idx.as<int32_t>(), W.rec.as<WinRow>(), W.dpath.as<unsigned char>(), A.v64.as<double>(),
        W.gval.as<double>(), otag, W.err.as<int>());
    FAIR_CUDA(cudaGetLastError());
    W.err_valid = true;
    W.uid += (uint64_t)nwin;
    *built = true;
    if (!want) return FAIR_OK;
    // on a cooperative grid, else on a cluster, the table in global memory; else in one
    // block, the table in its shared memory where it fits
    const size_t lv_bytes = 4 * (size_t)std::max<int32_t>(A.n, 1);
    if (W.lvtab.grow(lv_bytes)) {
        *built = false;
        return FAIR_OK;
    }
    FAIR_CUDA(cudaMemsetAsync(W.lvtab.p, 0, lv_bytes, s));
    if (!lvl_levels_grid<WR>(W, nord, C.dnlev.as<int>(), otag, s) &&
        !lvl_levels_cluster<WR>(W, nord, C.dnlev.as<int>(), otag, s)) {
        const bool smem = lv_bytes + 4096 <= optin;
        auto kern = smem ? k_lvl_levels<WR, true> : k_lvl_levels<WR, false>;
        if (smem)
            FAIR_CUDA(smem_allow(reinterpret_cast<const void *>(kern), lv_bytes));
        kern<<<1, 1024, smem ? lv_bytes : 0, s>>>(W.rec.as<WinRow>(), W.dpath.as<unsigned char>(),
                                                  W.idx.as<int32_t>(), nord, W.lvtab.as<int32_t>(), A.n,
                                                  W.lvl.as<int32_t>(), otag, C.dnlev.as<int>());
    }
    if (flow)
        k_lvl_tags<WR><<<sm_count() * 8, 256, 0, s>>>(W.rec.as<WinRow>(), nord, W.lvl.as<int32_t>(), otag);
    FAIR_CUDA(cudaGetLastError());
    return FAIR_OK;
}

// Builds (or takes from the cache of this sweep order) the level schedule and
// launches the level sweep. Returns FAIR_OK with *done = false (nothing
// launched) when its buffers cannot be had; the caller then runs the
// single-block kernel alone.
int lvl_sweep(const SweepDev &S, int dir, const RowStep *steps, const Box &box, bool *done,
              cudaStream_t s) {
    *done = false;
    SweepWork &W = *S.work;
    const DevCSR &A = *S.A;
    const int slot = dir > 0 ? 0 : 1;
    SweepWork::Levels &C = W.lev[slot];
    const bool cached = S.order_key != 0 && C.key == S.order_key && C.nord == S.nord;
    // orders drawn anew in every sweep get no levels, only (once per call) the
    // set-up's check for rows that repeat a column
    const bool want = S.order_key != 0 || env_int("FAIR_SWEEP_LEVELS_ALWAYS", 0);
    if (!want && W.err_valid) return FAIR_OK;
    if (!cached) {
        C.key = 0;
        const int32_t nord = S.nord;
        const int g = (int)std::min<int64_t>((nord + 255) / 256, (int64_t)sm_count() * 4);
        // the other direction's schedule of the same order, reversed
        const SweepWork::Levels &O = W.lev[1 - slot];
        if (S.order_key != 0 && O.key == S.order_key && O.nord == nord && W.err_valid) {
            if (O.use) {
                if (C.sched.grow(sizeof(RowStep) * (size_t)nord) || C.lptr.grow(8 * ((size_t)nord + 2)) ||
                    C.dnlev.grow(sizeof(int)))
                    return FAIR_OK;
                k_lvl_reverse<<<g, 256, 0, s>>>(O.sched.as<RowStep>(), O.lptr.as<int64_t>(), O.dnlev.as<int>(),
                                                nord, C.sched.as<RowStep>(), C.lptr.as<int64_t>(),
                                                C.dnlev.as<int>());
                FAIR_CUDA(cudaGetLastError());
            }
            C.nlev = O.nlev;
            C.entries = O.entries;
            C.use = O.use;
            C.grouped = O.grouped;
            C.key = S.order_key;
            C.nord = nord;
        }
    }
    if (S.order_key == 0 || C.key != S.order_key || C.nord != S.nord) {
        const int32_t nord = S.nord;
        const int g = (int)std::min<int64_t>((nord + 255) / 256, (int64_t)sm_count() * 4);
        int dev = 0, optin = 0;
        FAIR_CUDA(cudaGetDevice(&dev));
        FAIR_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
        // the widest window whose entries (a byte each) and stamps fit
        const int64_t row_max = std::max(A.max_row, 1);
        auto fits = [&](int wr) {
            return wr * row_max < (1 << kStampPosBits) && wr * row_max + wr * wr + 24 * wr + 1024 <= optin;
        };
        // (for the check alone the narrowest, the most windows at once: 2 sweeps in random
        // order, fan N=73, 84 angles, 15.42 ms in windows of 128, 15.09 in windows of 32)
        const int wr = want && fits(128) ? 128 : want && fits(64) ? 64 : 32;
        if (!fits(wr)) return FAIR_OK;
        if (W.lens.grow(4 * ((size_t)nord + 1)) || W.eoff.grow(8 * ((size_t)nord + 1)) ||
            W.rec.grow(sizeof(WinRow) * (size_t)nord) || W.lvl.grow(4 * (size_t)nord) ||
            W.cnt.grow(4 * ((size_t)nord + 1)) || W.err.grow(sizeof(int)) ||
            C.sched.grow(sizeof(RowStep) * (size_t)nord) || C.lptr.grow(8 * ((size_t)nord + 2)) ||
            C.dnlev.grow(sizeof(int)) || W.gsync.grow(4 * sizeof(int)))
            return FAIR_OK;
        FAIR_CUDA(cudaMemsetAsync(W.gsync.p, 0, 4 * sizeof(int), s));
        k_step_lengths<<<g, 256, 0, s>>>(steps, nord, W.lens.as<int32_t>());
        k_scan_excl<<<1, 1024, 0, s>>>(W.lens.as<int32_t>(), nord, nullptr, W.eoff.as<int64_t>());
        FAIR_CUDA(cudaMemsetAsync(W.err.p, 0, sizeof(int), s));
        FAIR_CUDA(cudaMemcpyAsync(&C.entries, W.eoff.as<int64_t>() + nord, sizeof(int64_t),
                                  cudaMemcpyDeviceToHost, s));
        FAIR_CUDA(cudaStreamSynchronize(s));
        const size_t ent = (size_t)C.entries;
        if (W.idx.grow(4 * std::max<size_t>(ent, 1))) return FAIR_OK;
        // the sweep without barriers needs a copy of the entries in step order with
        // their tags; the variables that pick a barrier sweep keep to it
        bool flow = want && S.order_key != 0 && env_int("FAIR_SWEEP_FLOW", 1) && !getenv("FAIR_SWEEP_CLUSTER") &&
                    !getenv("FAIR_SWEEP_GRID") && !getenv("FAIR_SWEEP_XMEM") &&
                    !W.gval.grow(8 * std::max<size_t>(ent, 1)) && !W.tag.grow(4 * std::max<size_t>(ent, 1)) &&
                    !W.pairs.grow(sizeof(XPair) * (size_t)std::max<int32_t>(A.n, 1));
        W.flow_slot = -1;
        W.lev[1 - slot].key = 0;  // its steps would point into the entries written now
        const size_t smem = (size_t)(wr * row_max);
        bool built = false;
        for (;;) {
            if (wr == 128) FAIR_TRY(lvl_build<128>(S, W, C, steps, smem, optin, want, flow, &built, s));
            else if (wr == 64) FAIR_TRY(lvl_build<64>(S, W, C, steps, smem, optin, want, flow, &built, s));
            else FAIR_TRY(lvl_build<32>(S, W, C, steps, smem, optin, want, flow, &built, s));
            if (built || !(W.gval.p || W.tag.p || W.pairs.p)) break;
            // no room for the level table beside the copies: levels without them
            flow = false;
            W.gval.release();
            W.tag.release();
            W.pairs.release();
        }
        if (!built || !want) return FAIR_OK;
        FAIR_CUDA(cudaMemsetAsync(W.cnt.p, 0, 4 * ((size_t)nord + 1), s));
        k_lvl_count<<<g, 256, 0, s>>>(W.lvl.as<int32_t>(), nord, W.cnt.as<int32_t>());
        k_scan_excl<<<1, 1024, 0, s>>>(W.cnt.as<int32_t>(), 0, C.dnlev.as<int>(), C.lptr.as<int64_t>());
        k_lvl_scatter<<<g, 256, 0, s>>>(steps, W.lvl.as<int32_t>(), nord, C.lptr.as<int64_t>(),
                                        W.cnt.as<int32_t>(), flow ? W.eoff.as<int64_t>() : nullptr,
                                        C.sched.as<RowStep>());
        FAIR_CUDA(cudaGetLastError());
        // levels pay when they hold several steps each (the ray orders: 30-80);
        // an order whose steps nearly all depend on the one before runs on the
        // single-block kernel
        int gerr = 0;
        FAIR_CUDA(cudaMemcpyAsync(&gerr, W.gsync.as<int>() + 2, sizeof(int), cudaMemcpyDeviceToHost, s));
        FAIR_CUDA(cudaMemcpyAsync(&C.nlev, C.dnlev.p, sizeof(int), cudaMemcpyDeviceToHost, s));
        FAIR_CUDA(cudaStreamSynchronize(s));
        if (gerr) {
            set_detail("Kaczmarz level set-up: a grid barrier timed out");
            return FAIR_ERR_CUDA;
        }
        if (flow) W.flow_slot = slot;
        C.grouped = flow;
        C.use = (int64_t)nord >= (int64_t)kMinStepsPerLevel * std::max(C.nlev, 1) ||
                env_int("FAIR_SWEEP_LEVELS_ALWAYS", 0);
        C.key = S.order_key;
        C.nord = nord;
    }
    if (!C.use) return FAIR_OK;
    const RowStep *sched = C.sched.as<RowStep>();
    const int64_t *lptr = C.lptr.as<int64_t>();
    const int *nlev = C.dnlev.as<int>();
    const int *err = W.err.as<int>();
    // warps per step: a long row (twice the mean, at most the longest) in 2
    // chunks of 32 entries per warp, at most 16 warps (a block): a warp's
    // FP64 instructions per step (64 cycles each) are on the level's critical
    // path. Measured (GB300, 10 sweeps of fan N=128 on the cluster, s): G = 1
    // 0.061, 2 0.041, 4 0.036, 8 0.038; 20 sweeps of fan N=512 symmetric on
    // the cooperative grid (s, blocks): G = 4 0.66 (26), 8 0.58 (51) / 0.52
    // (152), 16 0.47 (101) / 0.42 (152). FAIR_SWEEP_GROUP overrides (1, 2, 4,
    // 8 or 16).
    const double avg = S.nord > 0 ? (double)C.entries / S.nord : 0.0;
    int G = 1;
    while (G < 16 && 64.0 * G < std::min(2.0 * avg, (double)A.max_row)) G *= 2;
    const int Ge = env_int("FAIR_SWEEP_GROUP", 0);
    if (Ge == 1 || Ge == 2 || Ge == 4 || Ge == 8 || Ge == 16) G = Ge;
    if (W.gsync.grow(4 * sizeof(int))) return FAIR_OK;
    const double spl = C.nlev > 0 ? (double)S.nord / C.nlev : 1.0;
    const int32_t *col = C.grouped ? W.idx.as<int32_t>() : A.col.as<int32_t>();
    const double *val = C.grouped ? W.gval.as<double>() : A.v64.as<double>();
    if (C.grouped && W.flow_slot == slot) {
        // twice the warps of the barrier sweep: a warp's FP64 products lie on every
        // level's chain (G = 4, 8, 16: fan N=128 21.3, 20.3, 20.5 ms; N=512 108, 92,
        // 73 ms, two of its four sweeps with barriers)
        const int Gf = Ge == 1 || Ge == 2 || Ge == 4 || Ge == 8 || Ge == 16 ? Ge : std::min(16, 2 * G);
        int occ = 0;
        const bool wide = Gf == 16;
        auto kern = wide ? k_flow_sweep<2, 512, true> : k_flow_sweep<2, 512, false>;
        const int nb0 = env_int("FAIR_SWEEP_GRID_BLOCKS", 0);
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, 512, 0) == cudaSuccess && occ >= 1) {
            // room for two levels' steps in flight: more groups only poll (10 sweeps of fan
            // N=128, G = 8: 32 blocks 20.3 ms, 64 20.9, 152 22.0)
            const int room = (int)std::ceil(spl * 2.0 * Gf / 16.0);
            const int nb = std::min(nb0 > 0 ? nb0 : std::max(room, 1), occ * sm_count());
            auto launch = wide ? flow_launch<2, 512, true> : flow_launch<2, 512, false>;
            FAIR_TRY(launch(nb, sched, S.nord, col, val, W.tag.as<int32_t>(), W.pairs.as<XPair>(), S.x, A.n, box, Gf,
                            err, W.gsync.as<int>(), s, done));
            if (*done) return FAIR_OK;
        }
        cudaGetLastError();
    }
    FAIR_TRY((lvl_launch<2, 512>(S, sched, lptr, nlev, col, val, box, G, err, spl, s)));
    *done = true;
    return FAIR_OK;
}

}  // namespace

void SweepWork::release() {
    steps.release();
    lens.release();
    eoff.release();
    idx.release();
    rec.release();
    dpath.release();
    lvl.release();
    cnt.release();
    lvtab.release();
    err.release();
    tabs.release();
    gsync.release();
    gval.release();
    tag.release();
    pairs.release();
    bases.release();
    flow_slot = -1;
    for (Levels &L : lev) {
        L.sched.release();
        L.lptr.release();
        L.dnlev.release();
        L.key = 0;
        L.nord = L.nlev = 0;
        L.entries = 0;
        L.use = L.grouped = false;
    }
    tab_n = tab_blocks = 0;
    uid = 0;
    err_valid = false;
}

int kaczmarz_sweep(const SweepDev &S, int dir, cudaStream_t s) {
    if (S.nord <= 0) return FAIR_OK;
    SweepWork local;
    SweepWork &W = S.work ? *S.work : local;
    SweepDev SW = S;
    SW.work = &W;
    FAIR_TRY(W.steps.grow(sizeof(RowStep) * (size_t)S.nord));
    RowStep *steps = W.steps.as<RowStep>();
    const DevCSR &A = *S.A;
    int grid = (int)std::min<int64_t>(((int64_t)S.nord + 255) / 256, (int64_t)sm_count() * 8);
    k_sweep_schedule<<<grid, 256, 0, s>>>(S.ord, S.nord, dir, S.rand_rowprob ? 1 : 0, S.cumul, A.m,
                                          S.seed, S.ctr, A.rowptr.as<int64_t>(), S.b, S.nrA,
                                          S.omg, steps);
    FAIR_CUDA(cudaGetLastError());
    Box box;
    // a NaN bound leaves t unchanged unless t is NaN (MAX/MIN semantics); the
    // bound is then dropped, which differs only in the NaN payload
    box.mode = (S.bmode & 2) && !std::isnan(S.lb) ? 2 : 0;
    box.mode |= (S.bmode & 1) && !std::isnan(S.ub) ? 1 : 0;
    box.lb = S.lb;
    box.ub = S.ub;
    box.klb = host_key(S.lb);
    box.kub = host_key(S.ub);
    // the level sweep, and the single-block kernel behind it for a matrix
    // whose rows repeat a column (it runs only if the set-up said so);
    // FAIR_SWEEP_LEGACY=1 runs the single-block kernel alone
    bool leveled = false;
    const int *dup = nullptr;
    if (!env_int("FAIR_SWEEP_LEGACY", 0)) {
        FAIR_TRY(lvl_sweep(SW, dir, steps, box, &leveled, s));
        if (W.err_valid) dup = W.err.as<int>();
    }
    int dev = 0, optin = 0;
    FAIR_CUDA(cudaGetDevice(&dev));
    FAIR_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    const size_t need = sizeof(double) * (size_t)A.n;
    const bool smem = need + 4096 <= (size_t)optin;
    const int Wl = sweep_warps();
    const int oid = leveled ? 1 : 0;
    // entries per lane held in registers (longer rows finish in a loop)
    const int per_lane = (A.max_row + 32 * Wl - 1) / (32 * Wl);
    int st;
    switch (Wl) {
    case 1: st = per_lane <= 8 ? launch<1, 8>(SW, steps, smem, need, box, dup, oid, s)
                               : launch<1, 16>(SW, steps, smem, need, box, dup, oid, s);
        break;
    case 2: st = per_lane <= 8 ? launch<2, 8>(SW, steps, smem, need, box, dup, oid, s)
                               : launch<2, 16>(SW, steps, smem, need, box, dup, oid, s);
        break;
    case 4: st = per_lane <= 4 ? launch<4, 4>(SW, steps, smem, need, box, dup, oid, s)
                               : launch<4, 8>(SW, steps, smem, need, box, dup, oid, s);
        break;
    default: st = per_lane <= 2 ? launch<8, 2>(SW, steps, smem, need, box, dup, oid, s)
                                : launch<8, 4>(SW, steps, smem, need, box, dup, oid, s);
    }
    if (!S.work) {
        cudaStreamSynchronize(s);
        local.release();
    }
    return st;
}

}  // namespace fair
