// adjoint.cu -- reverse-mode adjoint of K unrolled SIRT/SART steps with box
// projection, for up to 16 right-hand sides sharing one matrix.
//
// Forward (AIRMs.f90:1089-1110, per right-hand side c with relaxation lam_c):
//   r_k = M^-1 (b - A x_k),  g_k = A' r_k,  z_k = x_k + (lam_c g_k) / D,
//   x_{k+1} = P(z_k) = max(min(z_k, ub), lb)   (the bounds present in opts)
// Reverse, for k = K-1 .. 0, starting from gx = dL/dx_K:
//   gz = gx * [P does not clamp z_k]
//   glam_c += <gz, g_k / D>
//   w = M^-1 A (D^-1 gz)        (w_i = 0 on empty rows, which b does not reach)
//   gb += lam_c w
//   gx = gz - lam_c A' w
// and dL/dx0 = gx after the last step. Checkpoints of x every ceil(sqrt(K))
// steps; each segment is recomputed forward (keeping x_k and g_k) before it
// is reversed, so memory is O(sqrt(K)) vectors and work is three forward
// sweeps of products.
//
// Vectors of the batch are interleaved ([row][NR], NR = 1, 4, 8 or 16) so that
// one gather loads every right-hand side of a column. Matrices whose columns
// (A) or rows (A') are an image run on the tiled copies (tl_multi_partials,
// tiled.cu: the gathered vectors staged in shared memory per tile) followed
// by row sums with the epilogue; others on the multi-vector row engine below.
// N = 256, 360 angles, 362 bins, 16 right-hand sides, FP32: a product takes
// 134 + 19 us (the row engine: 280 us); 101 x 101 fan, 180 angles, 3
// right-hand sides, FP64: 30 + 7 us (82 / 62).
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "fair_gpu_ext.h"
#include "fair_internal.cuh"
#include "rows.cuh"

namespace fair {

namespace {

constexpr int kG = 8;        // lanes per row of the multi-vector engine (one right-hand side)
constexpr int kRhsRows = 8;  // rows per chunk of the engine with right-hand sides across lanes

template <typename T, int NR>
__device__ __forceinline__ void load_row_vec(const T *__restrict__ p, T (&o)[NR]) {
#pragma unroll
    for (int r = 0; r < NR; ++r) o[r] = __ldg(p + r);
}

template <typename T, int NR, class Epi>
__device__ __forceinline__ void chunk_rows_multi(const int64_t *__restrict__ rowptr, int32_t m,
                                                 const int32_t *__restrict__ col,
                                                 const T *__restrict__ val,
                                                 const T *__restrict__ x, Epi &epi,
                                                 unsigned *sched) {
    constexpr int G = kG, R = 32 / G;
    const int lane = threadIdx.x & 31, g = lane / G, gl = lane % G;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int64_t nchunks = ((int64_t)m + 31) >> 5;
    for (int64_t ch = next_chunk(sched, 0, nwarps, lane); ch < nchunks;
         ch = next_chunk(sched, ch, nwarps, lane)) {
        const int64_t base = ch << 5;
        T mine[NR];
#pragma unroll
        for (int r = 0; r < NR; ++r) mine[r] = 0;
#pragma unroll 1
        for (int sub = 0; sub < 32; sub += R) {
            const int64_t row = base + sub + g;
            int64_t s = 0, e = 0;
            if (row < m) {
                s = __ldg(rowptr + row);
                e = __ldg(rowptr + row + 1);
            }
            T acc[NR];
#pragma unroll
            for (int r = 0; r < NR; ++r) acc[r] = 0;
            for (int64_t k = s + gl; k < e; k += G) {
                const int32_t c = __ldcs(col + k);
                const T v = __ldcs(val + k);
                T xv[NR];
                load_row_vec<T, NR>(x + (size_t)c * NR, xv);
#pragma unroll
                for (int r = 0; r < NR; ++r) acc[r] += v * xv[r];
            }
#pragma unroll
            for (int r = 0; r < NR; ++r) {
#pragma unroll
                for (int o = G / 2; o > 0; o >>= 1) acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], o);
                T t = __shfl_sync(0xffffffffu, acc[r], ((lane - sub) & (R - 1)) * G);
                if (lane >= sub && lane < sub + R) mine[r] = t;
            }
        }
        const int64_t row = base + lane;
        if (row < m) {
            const T y = epi.at(row);
#pragma unroll
            for (int c = 0; c < NR; ++c) epi.one(row, c, mine[c], y);
        }
    }
    finish_chunks(sched, nwarps, lane);
}

// The same products with the right-hand sides across the lanes (NR = 4, 8 or
// 16): lane l handles right-hand side l % NR of entry slot l / NR, so a warp
// step covers E = 32 / NR entries of one row and each entry's NR values of x
// are one contiguous run of NR x sizeof(T) bytes. The warp reads a row's
// entries 32 at a time (lane l loads entry l of the block: one coalesced load
// of columns and one of values, the next block's issued before the current
// one is used), hands each entry to its slot's lanes by shuffles, and keeps
// the block's 32 / E gathers of x in flight. The E slots are added by
// shuffles at the row's end and lanes 0..NR-1 apply the epilogue to the row's
// NR sums (Epi::one). A warp walks the kRhsRows rows of a chunk in turn;
// small chunks keep every warp of a persistent grid busy.
template <typename T, int NR, class Epi>
__device__ __forceinline__ void chunk_rows_rhs(const int64_t *__restrict__ rowptr, int32_t m,
                                               const int32_t *__restrict__ col,
                                               const T *__restrict__ val, const T *__restrict__ x,
                                               const Epi &epi, unsigned *sched) {
    static_assert(NR == 4 || NR == 8 || NR == 16, "4, 8 or 16 right-hand sides");
    constexpr int E = 32 / NR, STEPS = 32 / E, NA = 4, CR = kRhsRows;
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, slot = lane / NR, c = lane % NR;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int64_t nchunks = ((int64_t)m + CR - 1) / CR;
    for (int64_t ch = next_chunk(sched, 0, nwarps, lane); ch < nchunks;
         ch = next_chunk(sched, ch, nwarps, lane)) {
        const int64_t base = ch * CR;
        const int rows = (int)((int64_t)m - base < CR ? (int64_t)m - base : CR);
        for (int rr = 0; rr < rows; ++rr) {
            const int64_t row = base + rr;
            const int64_t s = __ldg(rowptr + row), e = __ldg(rowptr + row + 1);
            T acc[NA];
#pragma unroll
            for (int a = 0; a < NA; ++a) acc[a] = 0;
            int64_t kk = s + lane;
            int32_t cl = kk < e ? __ldcs(col + kk) : 0;
            T vl = kk < e ? __ldcs(val + kk) : (T)0;
            for (int64_t kb = s; kb < e; kb += 32) {
                // the next block's entries, loaded while this one is used
                const int64_t kn = kb + 32 + lane;
                const int32_t cn = kn < e ? __ldcs(col + kn) : 0;
                const T vn = kn < e ? __ldcs(val + kn) : (T)0;
                const int nb = (int)(e - kb < 32 ? e - kb : 32);
#pragma unroll
                for (int t = 0; t < STEPS; ++t) {
                    // steps past the row's end stay predicated: leaving the loop there
                    // (a warp-uniform break) keeps the gathers from issuing ahead, and
                    // measured FP32 throughput fell from 25 to 11 batch gradients/s
                    const int src = t * E + slot;
                    const int32_t cj = __shfl_sync(FULL, cl, src);
                    const T vj = __shfl_sync(FULL, vl, src);
                    if (src < nb) acc[t % NA] += vj * __ldg(x + (size_t)cj * NR + c);
                }
                cl = cn;
                vl = vn;
            }
            T v = (acc[0] + acc[1]) + (acc[2] + acc[3]);
#pragma unroll
            for (int o = 16; o >= NR; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
            if (lane < NR) epi.one(row, c, v, epi.at(row));
        }
    }
    finish_chunks(sched, nwarps, lane);
}

template <typename T>
__device__ __forceinline__ T boxT(T t, int bmode, T lb, T ub) {
    if (bmode & 1) t = t < ub || t != t ? t : ub;   // min(t, ub), the non-NaN wins
    if (bmode & 2) t = t > lb || t != t ? t : lb;   // max(t, lb)
    return t;
}

// Row (M) or column (D) weights that divide. An FP64 division is a sequence of
// 64-cycle instructions (N = 101 fan, 180 angles, 3 right-hand sides, 9 steps:
// 2.37 ms), so the product with the weight's reciprocal, formed in FP64 (1/0 = Inf),
// is taken (2.25 ms; the error against 64-bit sums is the same 1.2e-14 and, in
// FP32, 1.3e-7), and the division where that reciprocal overflows or is subnormal:
// inv holds 0 there.
template <typename T> struct Weights {
    const T *w, *inv;
    __device__ __forceinline__ T at(int64_t i) const { return inv[i]; }
    __device__ __forceinline__ T of(int64_t i, T y, T v, bool zero_if_empty = false) const {  // y = at(i)
        unsigned hi;
        if constexpr (sizeof(T) == 8) hi = (unsigned)__double2hiint(y);
        else hi = __float_as_uint(y);
        if (zero_if_empty && hi == (sizeof(T) == 8 ? 0x7FF00000u : 0x7F800000u)) return (T)0;
        return hi != 0u ? v * y : v / w[i];
    }
};
// forward pass 1: r = (b - A x) / M
template <typename T, int NR>
struct EpiFwdResid {
    const T *b;
    Weights<T> M;
    T *r;
    __device__ T at(int64_t i) const { return M.at(i); }
    __device__ void one(int64_t i, int c, T v, T y) const { r[i * NR + c] = M.of(i, y, b[i * NR + c] - v); }
};
// forward pass 2: g = A' r (kept when recording), x = P(x + lam g / D)
template <typename T, int NR>
struct EpiFwdUpdate {
    Weights<T> D;
    const T *lam;
    T *x, *gsave;
    T lb, ub;
    int bmode;
    __device__ T at(int64_t j) const { return D.w ? D.at(j) : (T)0; }
    __device__ void one(int64_t j, int c, T v, T y) const {
        T u = lam[c] * v;
        if (D.w) u = D.of(j, y, u);
        if (gsave) gsave[j * NR + c] = v;
        x[j * NR + c] = boxT<T>(x[j * NR + c] + u, bmode, lb, ub);
    }
};
// reverse, over A: w = (A t) / M (0 on empty rows), gb += lam w
template <typename T, int NR>
struct EpiAdjA {
    Weights<T> M;
    const T *lam;
    T *w, *gb;
    __device__ T at(int64_t i) const { return M.at(i); }
    __device__ void one(int64_t i, int c, T v, T y) const {
        const T wi = M.of(i, y, v, true);
        w[i * NR + c] = wi;
        gb[i * NR + c] += lam[c] * wi;
    }
};
// reverse, over A': gx = gz - lam A' w
template <typename T, int NR>
struct EpiAdjAT {
    const T *gz, *lam;
    T *gx;
    __device__ T at(int64_t) const { return (T)0; }
    __device__ void one(int64_t j, int c, T v, T) const { gx[j * NR + c] = gz[j * NR + c] - lam[c] * v; }
};

// (256, 4): up to 64 registers, so the 16 gathers of a block stay in flight
// without spills (measured: FP32 39 ms per 16-problem adjoint against 58 ms
// when the compiler chose 32 registers).
template <typename T, int NR, class Epi>
__global__ void __launch_bounds__(256, 4) k_multi(const int64_t *rowptr, int32_t m, const int32_t *col,
                                               const T *val, const T *x, Epi epi, unsigned *sched) {
    if constexpr (NR == 1)
        chunk_rows_multi<T, NR>(rowptr, m, col, val, x, epi, sched);
    else
        chunk_rows_rhs<T, NR>(rowptr, m, col, val, x, epi, sched);
}

// Row sums of the tiled products' partials (in row order) and the epilogue: a
// thread per row and 16 bytes of its NR values.
template <typename T, int NR, class Epi>
__global__ void __launch_bounds__(256) k_multi_rows(int32_t m, const int64_t *__restrict__ segbase,
                                                    const T *__restrict__ part, Epi epi) {
    constexpr int V = NR * sizeof(T) >= 16 ? 16 / (int)sizeof(T) : NR, L = NR / V;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < (int64_t)m * L;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = e / L;
        const int c0 = (int)(e % L) * V;
        T acc[V];
#pragma unroll
        for (int k = 0; k < V; ++k) acc[k] = 0;
        const int64_t k1 = segbase[i + 1];
        const T y = epi.at(i);
        for (int64_t k = segbase[i]; k < k1; ++k) {
            const T *p = part + (size_t)k * NR + c0;
            if constexpr (V == 4) {
                const float4 u = __ldcs(reinterpret_cast<const float4 *>(p));
                acc[0] += u.x; acc[1] += u.y; acc[2] += u.z; acc[3] += u.w;
            } else if constexpr (V == 2) {
                const double2 u = __ldcs(reinterpret_cast<const double2 *>(p));
                acc[0] += u.x; acc[1] += u.y;
            } else {
                acc[0] += __ldcs(p);
            }
        }
#pragma unroll
        for (int k = 0; k < V; ++k) epi.one(i, c0 + k, acc[k], y);
    }
}

// Elementwise reverse step: gz = gx * [P does not clamp z], t = gz / D,
// per-block partial sums of gz * g / D for every column (FP64).
template <typename T, int NR>
__global__ void __launch_bounds__(256) k_adj_mask(int64_t n, const T *x, const T *gk, Weights<T> D,
                                                  const T *lam, const T *gx, T *gz, T *t, int bmode,
                                                  T lb, T ub, double *partials) {
    __shared__ double sh[NR][8];
    double part = 0.0;
    const int64_t total = n * NR;
    // blockDim.x (256) and the grid stride are multiples of NR, so each thread
    // always handles the same column c = threadIdx.x % NR
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t j = e / NR;
        const int c = (int)(e % NR);
        T g = gk[e];
        T u = lam[c] * g;
        const T y = D.w ? D.at(j) : (T)0;
        if (D.w) u = D.of(j, y, u);
        T z = x[e] + u;
        bool pass = true;
        T zc = z;
        if (bmode & 1) { pass = pass && (z < ub); zc = z < ub ? z : ub; }
        if (bmode & 2) pass = pass && (zc > lb);
        T gzv = pass ? gx[e] : (T)0;
        gz[e] = gzv;
        t[e] = D.w ? D.of(j, y, gzv) : gzv;
        part += (double)gzv * (double)(D.w ? D.of(j, y, g) : g);
    }
    // reduce over the threads sharing a column: lanes c, c+NR, ... then warps
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o >= NR; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    if (lane < NR) sh[lane][wid] = part;
    __syncthreads();
    if (threadIdx.x < NR) {
        double s = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += sh[threadIdx.x][w];
        partials[(size_t)blockIdx.x * NR + threadIdx.x] = s;
    }
}

// glam of the steps of a segment: block k adds its step's partials, ge blocks x NR
// columns, to out[k][NR].
template <int NR>
__global__ void __launch_bounds__(256) k_adj_sums(const double *partials, int ge, double *out) {
    constexpr int L = 256 / NR;  // threads per column
    __shared__ double sh[256];
    const int c = threadIdx.x % NR, l = threadIdx.x / NR;
    const double *p = partials + (size_t)blockIdx.x * ge * NR;
    double acc = 0.0;
    for (int b = l; b < ge; b += L) acc += p[(size_t)b * NR + c];
    sh[threadIdx.x] = acc;
    for (int o = L / 2; o > 0; o >>= 1) {
        __syncthreads();
        if (l < o) sh[threadIdx.x] += sh[threadIdx.x + o * NR];
    }
    if (l == 0) out[(size_t)blockIdx.x * NR + c] = sh[c];
}

// x0 (column-major n x nrhs, or zeros) into the interleaved layout
template <typename T>
__global__ void k_interleave(const double *src, int64_t rows, int nrhs, int NRt, int c0, T *dst) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < rows * NRt;
         e += (int64_t)gridDim.x * blockDim.x) {
        int64_t i = e / NRt;
        int c = (int)(e % NRt);
        dst[e] = (src && c0 + c < nrhs && c < NRt) ? (T)src[(size_t)(c0 + c) * rows + i] : (T)0;
    }
}

template <typename T>
__global__ void k_deinterleave(const T *src, int64_t rows, int nrhs, int NRt, int c0, int ncols,
                               double *dst) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < rows * ncols;
         e += (int64_t)gridDim.x * blockDim.x) {
        int64_t i = e % rows;
        int c = (int)(e / rows);
        dst[(size_t)(c0 + c) * rows + i] = (double)src[i * NRt + c];
    }
}

template <typename T>
__global__ void k_weights(const double *a, int64_t n, T *w, T *inv) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        w[i] = (T)a[i];
        const T y = (T)(1.0 / a[i]), least = sizeof(T) == 8 ? (T)DBL_MIN : (T)FLT_MIN;
        inv[i] = w[i] != (T)0 && (isinf(y) || y < least) ? (T)0 : y;
    }
}

int egrid(int64_t n) {
    int64_t b = (n + 255) / 256;
    return (int)std::max<int64_t>(1, std::min<int64_t>(b, (int64_t)sm_count() * 4));
}

// Blocks of 8 warps for the chunks of m rows (32 rows per chunk for one
// right-hand side, kRhsRows for more), at most the resident blocks.
template <class K>
int mgrid(K kernel, int64_t m, int nr) {
    int occ = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, 256, 0);
    if (occ < 1) occ = 1;
    const int64_t rpc = nr == 1 ? 32 : kRhsRows;
    int64_t need = (((int64_t)m + rpc - 1) / rpc + 7) / 8;
    return (int)std::max<int64_t>(1, std::min<int64_t>((int64_t)sm_count() * occ, need));
}

// The handle's buffers (w_adj): kept between calls, each grown to what a call needs.
enum AdjBuf { AB_B, AB_X, AB_R, AB_GSEG, AB_XSEG, AB_CP, AB_GX, AB_GZ, AB_T, AB_W, AB_GB, AB_LAM, AB_M,
              AB_D, AB_PART, AB_STAGE, AB_SUM, AB_COUNT };

template <typename T, int NR>
int run_group(fair_csr h, const T *vA, const T *vAT, bool sart, const double *h_b,
              const double *h_x0, const double *h_gx, const double *h_lam, int nrhs, int c0,
              int ncols, int K, int bmode, double lb, double ub, const double *d_M64,
              const double *d_D64, double *h_xK, double *h_gb, double *h_gx0, double *h_glam) {
    DevCSR &A = h->A, &AT = h->AT;
    cudaStream_t s = h->stream;
    unsigned *sched = h->w_sched.as<unsigned>();
    constexpr int prec = sizeof(T) == 8 ? FAIR_PREC_F64 : FAIR_PREC_F32;
    const int64_t m = A.m, n = A.n;
    const int C = K > 0 ? (int)std::ceil(std::sqrt((double)K)) : 1;
    const int nseg = K > 0 ? (K + C - 1) / C : 0;
    static_assert(AB_COUNT <= sizeof(h->w_adj) / sizeof(h->w_adj[0]), "adjoint buffers");
    DevBuf *W = h->w_adj;
    const bool tiled1 = tl_multi_ready(A, prec, 1), tiled2 = tl_multi_ready(AT, prec, 2);
    const int ge = egrid(n * NR);
    for (int q : {AB_B, AB_R, AB_W, AB_GB}) FAIR_TRY(W[q].grow(sizeof(T) * m * NR));
    for (int q : {AB_X, AB_GX, AB_GZ, AB_T}) FAIR_TRY(W[q].grow(sizeof(T) * n * NR));
    FAIR_TRY(W[AB_CP].grow(sizeof(T) * n * NR * (size_t)(nseg + 1)));
    FAIR_TRY(W[AB_XSEG].grow(sizeof(T) * n * NR * (size_t)C));
    FAIR_TRY(W[AB_GSEG].grow(sizeof(T) * n * NR * (size_t)C));
    FAIR_TRY(W[AB_LAM].grow(sizeof(T) * NR));
    FAIR_TRY(W[AB_M].grow(sizeof(T) * m * 2));  // weights, then their reciprocals
    FAIR_TRY(W[AB_D].grow(sizeof(T) * n * 2));
    // the partial sums of glam, of all steps where they take no more than a vector (one
    // launch adds them up then), else of a segment; then glam of every step
    const bool all_sums = sizeof(double) * ge * (size_t)K <= sizeof(T) * (size_t)n;
    const size_t seg_sums = (size_t)ge * NR * (size_t)(all_sums ? std::max(K, 1) : C);
    FAIR_TRY(W[AB_SUM].grow(sizeof(double) * (seg_sums + (size_t)NR * (size_t)std::max(K, 1))));
    const int64_t segs = std::max<int64_t>(tiled1 ? A.tlm.nseg : 0, tiled2 ? AT.tlm.nseg : 0);
    FAIR_TRY(W[AB_PART].grow(sizeof(T) * NR * (size_t)segs));
    FAIR_TRY(W[AB_STAGE].grow(sizeof(double) * std::max<int64_t>(m, n) * ncols));
    T *b = W[AB_B].as<T>(), *x = W[AB_X].as<T>(), *r = W[AB_R].as<T>(), *gx = W[AB_GX].as<T>(),
      *gz = W[AB_GZ].as<T>(), *t = W[AB_T].as<T>(), *w = W[AB_W].as<T>(), *gb = W[AB_GB].as<T>(),
      *lam = W[AB_LAM].as<T>();
    double *stage = W[AB_STAGE].as<double>(), *sums = W[AB_SUM].as<double>(), *gl = sums + seg_sums;
    const size_t nNR = (size_t)n * NR, vecb = sizeof(T) * nNR;
    // inputs (stage is reused in stream order)
    auto put = [&](const double *src, int64_t rows, T *dst) -> int {
        if (src)
            FAIR_CUDA(cudaMemcpyAsync(stage, src + (size_t)c0 * rows, sizeof(double) * rows * ncols,
                                      cudaMemcpyHostToDevice, s));
        k_interleave<T><<<egrid(rows * NR), 256, 0, s>>>(src ? stage : nullptr, rows, ncols, NR, 0, dst);
        return FAIR_OK;
    };
    FAIR_TRY(put(h_b, m, b));
    FAIR_TRY(put(h_x0, n, x));
    FAIR_TRY(put(h_gx, n, gx));
    T lamh[NR];
    for (int c = 0; c < NR; ++c) lamh[c] = (T)(c < ncols ? h_lam[c0 + c] : 0.0);
    FAIR_CUDA(cudaMemcpyAsync(lam, lamh, sizeof(lamh), cudaMemcpyHostToDevice, s));
    auto weights = [&](const double *w64, int64_t rows, T *w) {
        k_weights<T><<<egrid(rows), 256, 0, s>>>(w64, rows, w, w + rows);
        return Weights<T>{w, w + rows};
    };
    const Weights<T> M = weights(d_M64, m, W[AB_M].as<T>());
    const Weights<T> D = sart ? weights(d_D64, n, W[AB_D].as<T>()) : Weights<T>{nullptr, nullptr};
    FAIR_CUDA(cudaMemsetAsync(gb, 0, sizeof(T) * m * NR, s));
    FAIR_CUDA(cudaGetLastError());
    const T tlb = (T)lb, tub = (T)ub;
    // epi(row, M v) over A (pass 1) or A' (pass 2)
    auto product = [&](int pass, const T *v, const auto &epi) -> int {
        using Epi = std::decay_t<decltype(epi)>;
        DevCSR &Q = pass == 1 ? A : AT;
        if (pass == 1 ? tiled1 : tiled2) {
            T *part = W[AB_PART].as<T>();
            FAIR_TRY(tl_multi_partials(Q, prec, NR, v, part, sched, s));
            k_multi_rows<T, NR, Epi><<<egrid((int64_t)Q.m * NR * 2), 256, 0, s>>>(
                Q.m, Q.tlm.segbase.as<int64_t>(), part, epi);
        } else {
            auto k = k_multi<T, NR, Epi>;
            k<<<mgrid(k, Q.m, NR), 256, 0, s>>>(Q.rowptr.as<int64_t>(), Q.m, Q.col.as<int32_t>(),
                                                pass == 1 ? vA : vAT, v, epi, sched);
        }
        FAIR_CUDA(cudaGetLastError());
        return FAIR_OK;
    };
    auto fwd_step = [&](T *gsave) -> int {
        FAIR_TRY(product(1, x, EpiFwdResid<T, NR>{b, M, r}));
        return product(2, r, EpiFwdUpdate<T, NR>{D, lam, x, gsave, tlb, tub, bmode});
    };
    // forward with checkpoints
    for (int k = 0; k < K; ++k) {
        if (k % C == 0)
            FAIR_CUDA(cudaMemcpyAsync(W[AB_CP].as<T>() + nNR * (k / C), x, vecb, cudaMemcpyDeviceToDevice, s));
        FAIR_TRY(fwd_step(nullptr));
    }
    auto get = [&](const T *src, int64_t rows, double *dst) -> int {
        k_deinterleave<T><<<egrid(rows * ncols), 256, 0, s>>>(src, rows, nrhs, NR, 0, ncols, stage);
        FAIR_CUDA(cudaMemcpyAsync(dst + (size_t)c0 * rows, stage, sizeof(double) * rows * ncols,
                                  cudaMemcpyDeviceToHost, s));
        FAIR_CUDA(cudaStreamSynchronize(s));
        return FAIR_OK;
    };
    if (h_xK) FAIR_TRY(get(x, n, h_xK));
    // reverse, one segment at a time; glam of each step stays on the device
    for (int seg = nseg - 1; seg >= 0; --seg) {
        const int k0 = seg * C, k1 = std::min(K, k0 + C);
        FAIR_CUDA(cudaMemcpyAsync(x, W[AB_CP].as<T>() + nNR * seg, vecb, cudaMemcpyDeviceToDevice, s));
        for (int k = k0; k < k1; ++k) {
            FAIR_CUDA(cudaMemcpyAsync(W[AB_XSEG].as<T>() + nNR * (k - k0), x, vecb,
                                      cudaMemcpyDeviceToDevice, s));
            FAIR_TRY(fwd_step(W[AB_GSEG].as<T>() + nNR * (k - k0)));
        }
        for (int k = k1 - 1; k >= k0; --k) {
            const T *xk = W[AB_XSEG].as<T>() + nNR * (k - k0);
            const T *gk = W[AB_GSEG].as<T>() + nNR * (k - k0);
            k_adj_mask<T, NR><<<ge, 256, 0, s>>>(n, xk, gk, D, lam, gx, gz, t, bmode, tlb, tub,
                                                 sums + (size_t)(all_sums ? k : k - k0) * ge * NR);
            FAIR_CUDA(cudaGetLastError());
            FAIR_TRY(product(1, t, EpiAdjA<T, NR>{M, lam, w, gb}));
            FAIR_TRY(product(2, w, EpiAdjAT<T, NR>{gz, lam, gx}));
        }
        if (!all_sums) k_adj_sums<NR><<<k1 - k0, 256, 0, s>>>(sums, ge, gl + (size_t)k0 * NR);
        else if (k0 == 0) k_adj_sums<NR><<<K, 256, 0, s>>>(sums, ge, gl);
        FAIR_CUDA(cudaGetLastError());
    }
    // outputs
    FAIR_TRY(get(gb, m, h_gb));
    FAIR_TRY(get(gx, n, h_gx0));
    std::vector<double> hgl((size_t)NR * K);
    if (K > 0) {
        FAIR_CUDA(cudaMemcpyAsync(hgl.data(), gl, sizeof(double) * hgl.size(), cudaMemcpyDeviceToHost, s));
        FAIR_CUDA(cudaStreamSynchronize(s));
    }
    double acc[NR] = {};
    for (int k = K - 1; k >= 0; --k)
        for (int c = 0; c < NR; ++c) acc[c] += hgl[(size_t)k * NR + c];
    for (int c = 0; c < ncols; ++c) h_glam[c0 + c] = acc[c];
    return FAIR_OK;
}

}  // namespace

void adjoint_release(fair_csr h) {
    cudaStreamSynchronize(h->stream);
    h->A.tlm.release();
    h->AT.tlm.release();
    for (DevBuf &b : h->w_adj) b.release();
}

int sirt_adjoint(fair_csr h, bool sart, int nrhs, const double *b, const double *x0, int K,
                 const double *lam, int bmode, double lb, double ub, const double *gx,
                 double *xK, double *gb, double *gx0, double *glam) {
    DevCSR &A = h->A, &AT = h->AT;
    cudaStream_t s = h->stream;
    FAIR_TRY(h->w_M.grow(sizeof(double) * ((size_t)A.m + 1)));
    FAIR_TRY(h->w_D.grow(sizeof(double) * ((size_t)A.n + 1)));
    FAIR_TRY(sirt_weights(A, AT, sart, h->w_M.as<double>(), h->w_D.as<double>(), s));
    const bool f32 = h->prec == FAIR_PREC_F32;
    if (f32) {
        FAIR_TRY(csr_make_lowprec(A, FAIR_PREC_F32, s));
        FAIR_TRY(csr_make_lowprec(AT, FAIR_PREC_F32, s));
    }
    // The tiled copies of the products (left unbuilt for matrices without an image)
    // where there is memory for them; without it the row engine runs, also when
    // they leave too little for the vectors.
    const Reclaim own(nullptr);  // what an allocation here may free is this function's to say
    if (K > 0) {
        int st = csr_make_tiled_multi(A, h->prec, 1, s);
        if (st == FAIR_OK) st = csr_make_tiled_multi(AT, h->prec, 2, s);
        if (st == FAIR_ERR_ALLOC) adjoint_release(h);
        else if (st != FAIR_OK) return st;
    }
    for (int c0 = 0; c0 < nrhs; c0 += 16) {
        const int nc = std::min(16, nrhs - c0);
        auto group = [&](auto nr) -> int {
            constexpr int NR = decltype(nr)::value;
            const double *M = h->w_M.as<double>(), *D = h->w_D.as<double>();
            if (f32)
                return run_group<float, NR>(h, A.v32.as<float>(), AT.v32.as<float>(), sart, b, x0, gx, lam,
                                            nrhs, c0, nc, K, bmode, lb, ub, M, D, xK, gb, gx0, glam);
            return run_group<double, NR>(h, A.v64.as<double>(), AT.v64.as<double>(), sart, b, x0, gx, lam,
                                         nrhs, c0, nc, K, bmode, lb, ub, M, D, xK, gb, gx0, glam);
        };
        auto run = [&]() -> int {
            if (nc == 1) return group(std::integral_constant<int, 1>());
            if (nc <= 4) return group(std::integral_constant<int, 4>());
            if (nc <= 8) return group(std::integral_constant<int, 8>());
            return group(std::integral_constant<int, 16>());
        };
        int st = run();
        if (st == FAIR_ERR_ALLOC) {  // all of a group's allocations come before its work
            adjoint_release(h);
            st = run();
        }
        if (st) return st;
    }
    return FAIR_OK;
}

}  // namespace fair
