// Dense FP64 inverse of the Schur complement B on the device.  The reference
// forms inv(B) with LAPACK (src/fluid-operators/laplacian.jl:118); B built
// through the nested-grid vort2flux is not symmetric (its relative asymmetry is
// 1e-6 … 1e-4 on the configurations tested), so a Cholesky factor would change
// the solution well above round-off.  This is Gauss–Jordan elimination with
// partial pivoting (the largest |value| of a column among the rows that have not
// been a pivot row), in place and without moving rows: the pivot row of column c
// is divided by the pivot, every other row takes its multiple, and column c
// becomes the column of the transformation.  With p_c the pivot row of column c
// the matrix ends as W with A⁻¹[c, p_c'] = W[p_c, c'].
//
// The elimination goes panel by panel.  A panel of w columns is eliminated by one
// block that holds it in registers, which leaves the panel's columns M of the
// transformation; the rest of the matrix takes the panel as one rank-w update
//     A ← A with rows J zeroed + M · A[J, :],   J = the panel's pivot rows.
// Up to n = 128 the panel is the whole matrix: one launch.  Where the registers
// hold fewer than 64 columns of all n rows, the same algorithm runs inside a copy
// of 64 columns, and the matrix takes all 64 as one update.
//
// What bounds it: the chain of columns, each three block barriers, a search by
// all threads and one pass over the panel (1.4 µs at n = 102, 1.7 at n = 314).
// Two launches per column on [B | I] (one block over n × 2n values in shared
// memory up to n = 112) took 521 µs at n = 102 and 3.06 ms at n = 314; this takes
// 140 µs and 0.69 ms.  In place but with the panel in shared memory: 250 µs and
// 1.38 ms, some 70 instructions per row and warp; in registers a value costs one
// multiply-add and half a shared load.
#include "ibpm_internal.cuh"

#include <algorithm>

namespace ibpm {

namespace {

constexpr int kGjBlock = 64;   // columns taken by the matrix as one update

// The largest key of a warp and the smallest row that has it.  |values| order as
// integers (key = bits + 1, 0 for no row), so three 32-bit reductions find it; row
// carries the value's sign in its last bit.
struct GjBest {
    unsigned hi, lo, row;
};
__device__ __forceinline__ GjBest gj_warp_best(GjBest b) {
    const unsigned hi = __reduce_max_sync(0xffffffffu, b.hi);
    const unsigned lo = __reduce_max_sync(0xffffffffu, b.hi == hi ? b.lo : 0u);
    const unsigned row = __reduce_min_sync(0xffffffffu, b.hi == hi && b.lo == lo ? b.row : 0xffffffffu);
    return {hi, lo, row};
}

// a[k] of a register array, k in [LO, HI) known at run time and the same for the
// warp, by bisection; a[k] ← 0.
template <int LO, int HI, int K>
__device__ __forceinline__ double gj_pick(double (&a)[K], int k) {
    if constexpr (HI - LO == 1) {
        const double v = a[LO];
        a[LO] = 0.0;
        return v;
    } else {
        constexpr int M = (LO + HI) / 2;
        if (k < M) return gj_pick<LO, M, K>(a, k);
        return gj_pick<M, HI, K>(a, k);
    }
}

// Eliminate columns [c0, c0 + w) of the matrix A (n rows, lda apart), w ≤ WC.
// Thread (g, x) holds column x of rows g·K … g·K + K − 1.  M (n × w) receives the
// transformation's columns, piv[c] the pivot rows, used[r] marks them (rows
// marked before take no part as pivots).  With `out` (w = n) the inverse itself
// is written there.
template <int WC, int T, int K>
__global__ void __launch_bounds__(T, 1) gj_panel_kernel(const double* A, int lda, int n, int c0, int w, double* M,
                                                        int* piv, unsigned char* used, double* out, int* info,
                                                        int col_base) {
    constexpr int G = T / WC;                  // groups of rows
    constexpr int KP = (K + 1) & ~1;           // rows of a group in fcol, for 16-byte loads
    __shared__ __align__(16) double fcol[G * KP];
    __shared__ double prow[WC];
    constexpr int NW = T / 32;
    __shared__ GjBest cand[NW];
    __shared__ unsigned char taken[G * KP];    // rows that are no longer (or never were) candidates
    __shared__ int spiv[WC];
    if (*info) return;                         // an earlier panel met a zero pivot
    const int tid = threadIdx.x, x = tid % WC, g = tid / WC;
    const int r0 = g * K;
    double a[K];
    {
        const double* src = A + (size_t)r0 * lda + c0 + x;
#pragma unroll
        for (int k = 0; k < K; ++k, src += lda) a[k] = r0 + k < n && x < w ? *src : 0.0;
    }
    for (int t = tid; t < G * KP; t += T) {
        const int r = t / KP * K + t % KP;
        taken[t] = t % KP >= K || r >= n || (used && used[r]);
    }
    for (int c = 0; c < w; ++c) {
        if (x == c) {                          // the owners of column c hand its values over
#pragma unroll
            for (int k = 0; k < K; ++k) {
                fcol[g * KP + k] = a[k];
                a[k] = 0.0;                    // column c starts again as the transformation's
            }
        }
        __syncthreads();
        GjBest b{0, 0, 0xffffffffu};
#pragma unroll
        for (int t = tid; t < G * KP; t += T) {
            const double f = fcol[t], v = fabs(f);
            const unsigned long long key = taken[t] || v != v ? 0ull : (unsigned long long)__double_as_longlong(v) + 1;
            const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;   // NaN is never a pivot
            if (hi > b.hi || (hi == b.hi && lo > b.lo)) b = {hi, lo, 2u * t + (f < 0.0)};
        }
        b = gj_warp_best(b);
        if ((tid & 31) == 0) cand[tid >> 5] = b;
        __syncthreads();
        b = gj_warp_best((tid & 31) < NW ? cand[tid & 31] : GjBest{0, 0, 0xffffffffu});
        if (b.hi == 0 && b.lo <= 1) {          // no row left, or the largest is zero: the same for every thread
            if (tid == 0) *info = col_base + c + 1;
            return;
        }
        const int at = (int)(b.row >> 1), gp = at / KP, kp = at % KP;   // the pivot row gp·K + kp
        if (g == gp) {                         // … divided by the pivot, which is the key and the sign
            const double mag = __longlong_as_double((long long)((((unsigned long long)b.hi << 32) | b.lo) - 1));
            const double v = gj_pick<0, K>(a, kp);
            prow[x] = (x == c ? 1.0 : v) / (b.row & 1 ? -mag : mag);
            if (x == 0) {
                spiv[c] = gp * K + kp;
                taken[at] = 1;
                fcol[at] = -1.0;               // in the pass below the cleared row becomes 0 + 1·prow
            }
        }
        __syncthreads();
        const double pr = prow[x];
#pragma unroll
        for (int k = 0; k < K; k += 2) {
            const double2 f = *reinterpret_cast<const double2*>(&fcol[g * KP + k]);
            a[k] = fma(-f.x, pr, a[k]);
            if (k + 1 < K) a[k + 1] = fma(-f.y, pr, a[k + 1]);
        }
        // fcol is written again by the next column's owners, after every
        // thread has read it
        if (c + 1 < w) __syncthreads();
    }
    __syncthreads();
    if (out) {
        // A⁻¹[c, p_x] = W[p_c, x]; fcol[r] ← the column whose pivot row r is
        for (int c = tid; c < w; c += T) fcol[spiv[c] / K * KP + spiv[c] % K] = (double)c;
        __syncthreads();
#pragma unroll
        for (int k = 0; k < K; ++k)
            if (r0 + k < n && x < w) out[(int)fcol[g * KP + k] * n + spiv[x]] = a[k];
        return;
    }
    {
        double* dst = M + (size_t)r0 * w + x;
#pragma unroll
        for (int k = 0; k < K; ++k, dst += w)
            if (r0 + k < n && x < w) *dst = a[k];
    }
    for (int c = tid; c < w; c += T) {
        piv[c] = spiv[c];
        used[spiv[c]] = 1;
    }
}

// The same elimination of one column c of the n × w panel M in global memory, for
// n beyond the registers: the pivot (one block; its row divided by it into prow,
// column c saved into fcol and cleared), then the multiples.
__global__ void __launch_bounds__(1024) gj_column_kernel(double* M, int n, int w, int c, double* fcol, double* prow,
                                                         int* piv, unsigned char* used, int* info, int col_base) {
    __shared__ double bv[32];
    __shared__ int bi[32];
    if (*info) return;
    const int tid = threadIdx.x, lane = tid & 31;
    double best = 0.0;
    int row = n;
    for (int r = tid; r < n; r += 1024) {
        const double v = M[(size_t)r * w + c];
        fcol[r] = v;
        M[(size_t)r * w + c] = 0.0;
        if (!used[r] && (fabs(v) > fabs(best) || (row == n && v == 0.0))) { best = v; row = r; }
    }
    for (int pass = 0; pass < 2; ++pass) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const double o = __shfl_xor_sync(0xffffffffu, best, off);
            const int oi = __shfl_xor_sync(0xffffffffu, row, off);
            if (fabs(o) > fabs(best) || (fabs(o) == fabs(best) && oi < row)) { best = o; row = oi; }
        }
        if (pass == 0) {
            if (lane == 0) { bv[tid >> 5] = best; bi[tid >> 5] = row; }
            __syncthreads();
            best = bv[lane];
            row = bi[lane];
        }
    }
    if (row >= n || best == 0.0) {
        if (tid == 0) *info = col_base + c + 1;
        return;
    }
    if (tid < w) {
        const double v = (tid == c ? 1.0 : M[(size_t)row * w + tid]) / best;
        prow[tid] = v;
        M[(size_t)row * w + tid] = v;
    }
    if (tid == 0) { piv[c] = row; used[row] = 1; }
}

__global__ void gj_multiples_kernel(double* M, int n, int w, int c, const double* __restrict__ fcol,
                                    const double* __restrict__ prow, const int* piv, const int* info) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (*info || t >= (long long)n * w) return;
    const int r = (int)(t / w), col = (int)(t % w);
    if (r != piv[c]) M[t] = fma(-fcol[r], prow[col], M[t]);
}

// P ← columns [c0, c0 + w) of A.
__global__ void gj_take_kernel(const double* A, int n, int c0, int w, double* P) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < (long long)n * w) P[t] = A[(size_t)(t / w) * n + c0 + t % w];
}

// R = A[J, :] over nc columns, those rows of A zeroed.  The panel's own columns
// [c0, c0 + w) start from zero with R = I, so the update leaves M in them.
__global__ void __launch_bounds__(256) gj_rows_kernel(double* A, int lda, int nc, int n, int c0, int w,
                                                      const int* __restrict__ piv, double* R, const int* info) {
    if (*info) return;
    const int col = blockIdx.x * 32 + (threadIdx.x & 31), t = threadIdx.x >> 5;
    if (col >= nc) return;
    if (col >= c0 && col < c0 + w) {
        for (int r = t; r < n; r += 8) A[(size_t)r * lda + col] = 0.0;
        for (int c = t; c < w; c += 8) R[(size_t)c * nc + col] = col - c0 == c ? 1.0 : 0.0;
        return;
    }
#pragma unroll 8
    for (int c = t; c < w; c += 8) {
        const size_t at = (size_t)piv[c] * lda + col;
        R[(size_t)c * nc + col] = A[at];
        A[at] = 0.0;
    }
}

// A += M · R (n×w times w×nc), 64×64 tiles per block, k in chunks of 32.
__global__ void __launch_bounds__(256) gj_update_kernel(double* A, int lda, int nc, int n, int w,
                                                        const double* __restrict__ M, const double* __restrict__ R,
                                                        const int* info) {
    if (*info) return;
    __shared__ double Xs[64][33];
    __shared__ double Rs[32][65];
    const int r0 = blockIdx.y * 64, col0 = blockIdx.x * 64;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;   // 16 × 16 threads, 4 × 4 outputs each
    double acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = 0.0;
    for (int k0 = 0; k0 < w; k0 += 32) {
        for (int t = threadIdx.x; t < 64 * 32; t += 256) {
            const int rr = t / 32, kk = t % 32;
            Xs[rr][kk] = (r0 + rr < n && k0 + kk < w) ? M[(size_t)(r0 + rr) * w + k0 + kk] : 0.0;
            const int k2 = t / 64, cc = t % 64;
            Rs[k2][cc] = (k0 + k2 < w && col0 + cc < nc) ? R[(size_t)(k0 + k2) * nc + col0 + cc] : 0.0;
        }
        __syncthreads();
        const int km = min(32, w - k0);
#pragma unroll 8
        for (int kk = 0; kk < km; ++kk) {
            double xa[4], rb[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) xa[a] = Xs[ty * 4 + a][kk];
#pragma unroll
            for (int b = 0; b < 4; ++b) rb[b] = Rs[kk][tx + 16 * b];
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) acc[a][b] = fma(xa[a], rb[b], acc[a][b]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const int r = r0 + ty * 4 + a;
        if (r >= n) continue;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int col = col0 + tx + 16 * b;
            if (col < nc) A[(size_t)r * lda + col] += acc[a][b];
        }
    }
}

// W ← A, no row used.
__global__ void gj_start_kernel(const double* A, double* W, unsigned char* used, int n) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < (long long)n * n) W[t] = A[t];
    if (t < n) used[t] = 0;
}

// A[c, piv[k]] ← W[piv[c], k]
__global__ void gj_finish_kernel(const double* W, double* A, const int* __restrict__ piv, int n, const int* info) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (*info || t >= (long long)n * n) return;
    const int c = (int)(t / n), k = (int)(t % n);
    A[(size_t)c * n + piv[k]] = W[(size_t)piv[c] * n + k];
}

// The panel width for n > 128: 256 threads hold (256 / w) · K rows of w columns,
// K ≤ 88 doubles of registers (80 at w = 4: fcol, n doubles, must fit the static
// 48 KB of shared memory).  0 from n = 5121 on: columns one by one in global
// memory.  Fewer threads with more rows each are faster: a column's fixed costs
// (barriers, the scan of the candidates) grow with the warps; 1024 threads took
// 3.1 µs per column at n = 102.
int gj_width(int n) {
    for (int w = kGjBlock; w >= 8; w /= 2)
        if ((256 / w) * 88 >= n) return w;
    return 64 * 80 >= n ? 4 : 0;
}

// Work layout for n > 128: the matrix (n×n), M (n×64), R (64×n), inside a block
// Mi (n×64), Ri (64×64), then piv (n ints) and used (n bytes).
struct GjWork {
    double *A, *M, *R, *Mi, *Ri;
    int* piv;
    unsigned char* used;
    size_t doubles;
    GjWork(double* base, int n) {
        const size_t W = kGjBlock, nn = (size_t)n;
        A = base;
        M = A + nn * nn;
        R = M + nn * W;
        Mi = R + nn * W;
        Ri = Mi + nn * W;
        piv = reinterpret_cast<int*>(Ri + W * W);
        used = reinterpret_cast<unsigned char*>(piv + nn);
        doubles = nn * nn + 3 * nn * W + W * W + (5 * nn + 7) / 8;
    }
};

// The panel kernel of the fewest rows per thread that holds n rows.  Each count is
// a kernel of its own, so there are three per width: 52 fits the registers (204 to
// 216 of 255), 80 spills 7 to 12 doubles a thread, 88 some 50, for which a width
// reaches a tenth further before the next one halves it.  52 and 80 hold the 102
// components of the pitching plate and the 314 of the 200² cylinder closely; other
// sizes pay for the rows they leave empty, since a column passes over all K.
template <int WC>
cudaError_t gj_panel_w(const double* A, int lda, int n, int c0, int w, double* M, int* piv, unsigned char* used,
                       int* info, int col_base, cudaStream_t st) {
    constexpr int G = 256 / WC;
#define GJ_GO(K) gj_panel_kernel<WC, 256, K><<<1, 256, 0, st>>>(A, lda, n, c0, w, M, piv, used, nullptr, info, col_base)
    if (n <= 52 * G) GJ_GO(52);
    else if (n <= 80 * G) GJ_GO(80);
    else if constexpr (WC > 4) GJ_GO(88);
    else return cudaErrorInvalidValue;
#undef GJ_GO
    return cudaGetLastError();
}

cudaError_t gj_panel(int WC, const double* A, int lda, int n, int c0, int w, double* M, int* piv, unsigned char* used,
                     int* info, int col_base, cudaStream_t st) {
    switch (WC) {
        case 64: return gj_panel_w<64>(A, lda, n, c0, w, M, piv, used, info, col_base, st);
        case 32: return gj_panel_w<32>(A, lda, n, c0, w, M, piv, used, info, col_base, st);
        case 16: return gj_panel_w<16>(A, lda, n, c0, w, M, piv, used, info, col_base, st);
        case 8: return gj_panel_w<8>(A, lda, n, c0, w, M, piv, used, info, col_base, st);
        default: return gj_panel_w<4>(A, lda, n, c0, w, M, piv, used, info, col_base, st);
    }
}

}  // namespace

size_t gj_work_doubles(int n) { return n <= 128 ? 1 : GjWork(nullptr, n).doubles; }

cudaError_t launch_gj_inverse(double* A, int n, double* work, int* info, cudaStream_t st) {
    if (n < 1) return cudaErrorInvalidValue;
    cudaError_t e = cudaMemsetAsync(info, 0, sizeof(int), st);
    if (e != cudaSuccess) return e;
    if (n <= 128) {
#define GJ_ALL(WC, T, K) gj_panel_kernel<WC, T, K><<<1, T, 0, st>>>(A, n, n, 0, n, nullptr, nullptr, nullptr, A, info, 0)
        if (n <= 32) GJ_ALL(32, 128, 8);
        else if (n <= 64) GJ_ALL(64, 256, 16);
        else if (n <= 104) GJ_ALL(128, 256, 52);
        else GJ_ALL(128, 256, 64);
#undef GJ_ALL
        return cudaGetLastError();
    }
    const GjWork k(work, n);
    const int WC = gj_width(n);
    const unsigned all = (unsigned)(((long long)n * n + 255) / 256);
    gj_start_kernel<<<all, 256, 0, st>>>(A, k.A, k.used, n);
    for (int j0 = 0; j0 < n; j0 += kGjBlock) {
        const int w = std::min(kGjBlock, n - j0);
        int* piv = k.piv + j0;
        if (WC == kGjBlock) {
            if ((e = gj_panel(WC, k.A, n, n, j0, w, k.M, piv, k.used, info, j0, st)) != cudaSuccess) return e;
        } else {
            const unsigned each = (unsigned)(((long long)n * w + 255) / 256);
            gj_take_kernel<<<each, 256, 0, st>>>(k.A, n, j0, w, k.M);
            for (int c = 0; WC == 0 && c < w; ++c) {
                gj_column_kernel<<<1, 1024, 0, st>>>(k.M, n, w, c, k.Mi, k.Ri, piv, k.used, info, j0);
                gj_multiples_kernel<<<each, 256, 0, st>>>(k.M, n, w, c, k.Mi, k.Ri, piv, info);
            }
            for (int c0 = 0; WC > 0 && c0 < w; c0 += WC) {
                const int v = std::min(WC, w - c0);
                if ((e = gj_panel(WC, k.M, w, n, c0, v, k.Mi, piv + c0, k.used, info, j0 + c0, st)) != cudaSuccess) return e;
                gj_rows_kernel<<<(w + 31) / 32, 256, 0, st>>>(k.M, w, w, n, c0, v, piv + c0, k.Ri, info);
                gj_update_kernel<<<dim3((w + 63) / 64, (n + 63) / 64), 256, 0, st>>>(k.M, w, w, n, v, k.Mi, k.Ri, info);
            }
        }
        gj_rows_kernel<<<(n + 31) / 32, 256, 0, st>>>(k.A, n, n, n, j0, w, piv, k.R, info);
        gj_update_kernel<<<dim3((n + 63) / 64, (n + 63) / 64), 256, 0, st>>>(k.A, n, n, n, w, k.M, k.R, info);
    }
    gj_finish_kernel<<<all, 256, 0, st>>>(k.A, A, k.piv, n, info);
    return cudaGetLastError();
}

}  // namespace ibpm
