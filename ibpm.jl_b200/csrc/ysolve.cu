// The y-direction of a Poisson-type solve x = S((S b) ./ M .* scale), S the
// 2-D DST-I (src/fluid-operators/dst-inversion.jl:39-50, laplacian.jl:24-76).
//
// After the x-transform every x-mode k is an independent problem along y.  The
// operator the DST-I diagonalises is the 5-point stencil with zero Dirichlet
// edges (Δ: 4u − Σ neighbours; A: u + c(4u − Σ neighbours)), so mode k of it is
// the constant-coefficient tridiagonal system, j = 1 … ny−1, u_0 = u_ny = 0,
//     p u_j + c (2 u_j − u_{j−1} − u_{j+1}) = f_j,
//     p = λ (Δ, c = 1)  or  1 + c λ (A),   λ = 4 sin²(πk/(2nx)),
// and solving it directly gives what transform, divide and transform back
// give.  With r the root in (0, 1) of c (1 − r)² = p r it factors into two
// first-order recursions,
//     v_j = g_j + r v_{j−1}   (g = f, rising j),      w_j = v_j + r w_{j+1}   (falling j),
//     u = κ w,  κ = r / c = 1 / (c + p/2 + √(p c + p²/4)),
// exact in the interior and at u_ny = 0; a source g_0 = −w_0 (1−r²)/(1−r^{2ny})
// in row 0 (w_0 computed with g_0 = 0) makes u_0 = 0 too.  Every term is a sum of products of
// like signs except that last correction, and λ is formed without
// cancellation: against an extended-precision solve the error is 1e-15 … 1e-14
// where dividing by −2(cos + cos − 2) leaves 1e-12 at 512² and 2e-11 at 2048².
//
// What bounds it: one read and one write of the field (a few dozen operations
// per point); at 512² the latency of one load-scan-store chain.  The
// transform-divide-transform kernel this replaces went through shared memory
// ten times per point; the step of 512² x 5 levels went from 324 to 237 µs with
// this one (six such launches), that of 1024² x 5 from 1085 to 703 µs.
#include "ibpm_internal.cuh"

namespace ibpm {

namespace {

// b^e for e ≥ 0 by squaring
__device__ __forceinline__ double pow_int(double b, int e) {
    double p = 1.0;
    while (e) {
        if (e & 1) p *= b;
        b *= b;
        e >>= 1;
    }
    return p;
}

// One CTA solves TX neighbouring modes over all rows.  Rows 0 … ny−1 (row 0 the
// boundary) are cut into nc = ny / C chunks; thread (c, x) holds the C rows of
// chunk c of mode i0 + x in registers.  Its local recursions give the chunk's
// last v and first w; LPM lanes per mode (E chunks each) combine those over the
// chunks in a shuffle scan, which also yields w_0 and so the boundary source;
// each thread then adds its carries and finishes.  TX consecutive values of a
// row are whole 32-byte sectors.  The constants of a mode depend on the
// problem only and are formed before the dependency wait.
//
// SRC, how f is formed:
//   YSRC_DATA    read from the slab, solved in place
//   YSRC_EDGES   the x-spectrum of apply_bc!(e) of the slab's level (BtSynth),
//                into `out` (same slab map): with S(i, k) = 2 sin(π i k / nx),
//                f(k, j) = S(1, k) e_L(j) + S(nx−1, k) e_R(j)
//                        + [j = 1] Σ_i S(i, k) e_B(i) + [j = ny−1] Σ_i S(i, k) e_T(i)
//   YSRC_BOTH    in_scale × the slab's rows [in0, in1) plus, where hat is given,
//                the edges with their bottom and top sums already formed; only
//                rows [out0, out1) (or the bodies', rowbox) stored
//   YSRC_UNIT    the x-spectrum of C'E' e_kk of force component col0 + batch
//                (B_times!, laplacian.jl:162), 14×14 values around its point
// Resident CTAs per SM the register budget is set for: 1024 threads of at most
// 64 registers, or 768 of 80 where a thread holds 16 rows.
template <int C, int THREADS> constexpr int ys_min_blocks() {
    return THREADS > 512 ? 1 : (C > 8 ? 768 : 1024) / THREADS;
}

template <class T, int C, int TX, int LPM, int E, int SRC>
__global__ void __launch_bounds__(TX * LPM * E, ys_min_blocks<C, TX * LPM * E>())
    y_solve_kernel(T* data, SlabMap map, Geom g, const __grid_constant__ SpecParams sp, T* out,
                   const __grid_constant__ YSource ys) {
    constexpr int LC = LPM * E + 1;                      // chunk pitch of the exchange arrays (odd)
    __shared__ double sV[TX * LC], sW[TX * LC];
    __shared__ double sC[4 * TX];                        // r, κ·scale, 1/(1−r^{2ny}), 1−r² of each mode
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* sn = reinterpret_cast<double*>(smem_raw);    // edges, unit: sin(π t/nx), t < nx
    const int P = g.P, n1 = g.n1, nx = g.nx, nc = g.ny / C;
    const int tid = threadIdx.x, x = tid % TX, c = tid / TX;
    const bool own = c < nc;                             // the block is padded to whole warps
    const int i0 = blockIdx.x * TX, col = i0 + x;
    const int lev = map.level(blockIdx.y), bt = map.batch(blockIdx.y);
    const long long soff = map.off(blockIdx.y);
    const int o0 = (c * C - 1) * P + col;                // row c·C of the grid is slab row c·C − 1

    if (tid < TX) {
        const bool delta = sp.mode == SPEC_DELTA;
        const double* md = sp.mden ? sp.mden + (long long)bt * 9 : nullptr;
        const double cs = delta ? 1.0 : (md ? md[8] / md[lev] : sp.dt / sp.den[lev]);   // c of the stencil
        const double s = sinpi((double)(col + 1) / (double)(2 * nx));
        const double lam = 4.0 * s * s;
        const double p = delta ? lam : fma(cs, lam, 1.0);
        const double kap = 1.0 / (cs + 0.5 * p + sqrt(p * (cs + 0.25 * p)));
        const double r = cs * kap;
        sC[tid] = r;
        sC[TX + tid] = kap * sp.scale;
        sC[2 * TX + tid] = 1.0 / (1.0 - pow_int(r * r, g.ny));
        sC[3 * TX + tid] = 1.0 - r * r;
    }
    if constexpr (SRC == YSRC_UNIT || SRC == YSRC_EDGES)
        for (int t = tid; t < nx; t += blockDim.x) sn[t] = ys.edges.sx[t];
    pdl_wait();
    pdl_trigger();

    // lane l of mode sm in the scan over the chunks
    const int sm = tid / LPM, l = tid % LPM;
    const bool scans = sm < TX;                          // whole warps
    auto sinpix = [&](int t) -> double { return t < nx ? sn[t] : -sn[t - nx]; };   // 0 ≤ t < 2 nx
    double v[C];
    if constexpr (SRC == YSRC_DATA || SRC == YSRC_BOTH) {
        const T* src = data + soff;
        T raw[C];
#pragma unroll
        for (int i = 0; i < C; ++i) {
            const int j = c * C + i - 1;                 // slab row
            const bool in = SRC == YSRC_DATA ? j >= 0 : j >= ys.in0 && j < ys.in1;
            raw[i] = (own && in && col < n1) ? src[o0 + i * P] : T(0);
        }
        __syncthreads();                                 // sC, sn, while the loads are in flight
#pragma unroll
        for (int i = 0; i < C; ++i) v[i] = SRC == YSRC_DATA ? (double)raw[i] : ys.in_scale * (double)raw[i];
    } else {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < C; ++i) v[i] = 0.0;
    }
    // S(1, k) of the mode; S(nx−1, k) = (−1)^{k+1} S(1, k)
    auto side = [&](const double* eL, const double* eR, double s1) {
        const double sr = col & 1 ? -1.0 : 1.0;          // k = col + 1
#pragma unroll
        for (int i = 0; i < C; ++i) {
            const int j = c * C + i - 1;
            if (own && j >= 0) v[i] = fma(s1, fma(sr, __ldg(&eR[j]), __ldg(&eL[j])), v[i]);
        }
    };
    if constexpr (SRC == YSRC_BOTH) {
        if (ys.hat) {
            const double* e = ys.hat + (long long)bt * (2 * nx + 2 * g.ny);
            side(e + 2 * nx, e + 2 * nx + g.ny, 2.0 * __ldg(&ys.edges.sx[min(col + 1, nx - 1)]));
            if (c == 0) v[1] += e[col];
            if (c == nc - 1) v[C - 1] += e[nx + col];
        }
    }
    if constexpr (SRC == YSRC_EDGES) {
        const int ep = (2 * n1 + 2 * g.n2 + 3) & ~3;
        const double* e = ys.edges.e + ((long long)bt * g.mg + lev) * ep;
        const int k = col + 1, nx2 = 2 * nx;
        // this thread's share of the sine sums of the bottom and top rows
        if (own) {
            double pb = 0.0, pt = 0.0;
            int t = ((c + 1) * k) % nx2;
            const int dt = (nc * k) % nx2;
#pragma unroll 4
            for (int i = c; i < n1; i += nc) {
                const double sv = sinpix(t);
                pb = fma(sv, __ldg(&e[i]), pb);
                pt = fma(sv, __ldg(&e[n1 + i]), pt);
                t += dt;
                if (t >= nx2) t -= nx2;
            }
            sV[x * LC + c] = pb;
            sW[x * LC + c] = pt;
        }
        side(e + 2 * n1, e + 2 * n1 + g.n2, 2.0 * sinpix(k % nx2));
        __syncthreads();
        if (scans) {                                     // sums over the chunks
            double b = 0.0, tt = 0.0;
#pragma unroll
            for (int q = l; q < LPM * E; q += LPM) {
                b += q < nc ? sV[sm * LC + q] : 0.0;
                tt += q < nc ? sW[sm * LC + q] : 0.0;
            }
#pragma unroll
            for (int off = LPM / 2; off > 0; off >>= 1) {
                b += __shfl_xor_sync(0xffffffffu, b, off);
                tt += __shfl_xor_sync(0xffffffffu, tt, off);
            }
            if (l == 0) {
                sV[sm * LC] = 2.0 * b;
                sW[sm * LC] = 2.0 * tt;
            }
        }
        __syncthreads();
        if (c == 0) v[1] += sV[x * LC];
        if (c == nc - 1) v[C - 1] += sW[x * LC];
        __syncthreads();
    }
    if constexpr (SRC == YSRC_UNIT) {
        __shared__ double src[14][15];                   // [row][column] of the box
        const int kk = ys.col0 + bt, comp = kk / ys.nb, pt = kk % ys.nb;
        const int bx = ys.bidx[pt], by = ys.bidx[ys.nb + pt];
        const double* wt = ys.w + (long long)kk * 169;
        for (int t = tid; t < 196; t += blockDim.x) {
            const int da = t % 14, db = t / 14;
            // Γ[gi, gj] = (qx[gi+1, gj] − qx[gi+1, gj+1]) + (qy[gi+1, gj+1] − qy[gi, gj+1]) of the window's
            // weights (rot!, curl.jl:22-34), gi = bx − 7 + da, gj = by − 7 + db
            auto at = [&](int l2, int m2) -> double {
                return l2 >= 0 && l2 < 13 && m2 >= 0 && m2 < 13 ? wt[l2 * 13 + m2] : 0.0;
            };
            double val;
            if (comp == 0) val = at(da, db - 1) - at(da, db);
            else val = at(da, db) - at(da - 1, db);
            const int gi = bx - 7 + da, gj = by - 7 + db;
            src[db][da] = gi >= 1 && gi <= n1 && gj >= 1 && gj <= g.n2 ? val : 0.0;
        }
        __syncthreads();
        const int k = col + 1, nx2 = 2 * nx, j0 = by - 7;    // grid row of the box's first row
        if (own && c * C + C > j0 && c * C < j0 + 14) {
            int t = (int)(((long long)max(bx - 7, 0) * k) % nx2);
            const int a0 = max(7 - bx, 0);               // gi = 0 or below: no values there
            for (int da = a0; da < 14; ++da) {
                const double sv = 2.0 * sinpix(t);
#pragma unroll
                for (int i = 0; i < C; ++i) {
                    const int db = c * C + i - j0;
                    if (db >= 0 && db < 14) v[i] = fma(sv, src[db][da], v[i]);
                }
                t += k;
                if (t >= nx2) t -= nx2;
            }
        }
    }

    // local recursions: v with zero carry, and the chunk's first w
    const double r = sC[x];
#pragma unroll
    for (int i = 1; i < C; ++i) v[i] = fma(r, v[i - 1], v[i]);
    double w = v[C - 1];
    if (own) sV[x * LC + c] = w;
#pragma unroll
    for (int i = C - 2; i >= 0; --i) w = fma(r, w, v[i]);
    if (own) sW[x * LC + c] = w;
    __syncthreads();

    // over the chunks: A_c, the carry into the first row of chunk c, rising;
    // B_c, its first w, falling; then the boundary source's part of both:
    // g_0 R^c to the carry and −w_0 (R^{c+1} − R^{2nc−c−1})/(1 − R^{2nc}) to
    // the first w of chunk c+1, R = r^C
    if (scans) {
        const double rs = sC[sm];
        double R = rs, K = 1.0, qq = rs * rs;            // K = Σ_{i<C} r^{2i}
#pragma unroll
        for (int s = 1; s < C; s <<= 1) {
            K = fma(K, qq, K);
            qq *= qq;
            R *= R;
        }
        double A[E], B[E], inc = 0.0;
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const int cc = l * E + e;
            A[e] = cc < nc ? rs * sV[sm * LC + cc] : 0.0;
            B[e] = cc < nc ? sW[sm * LC + cc] : 0.0;
            inc = fma(R, inc, A[e]);
        }
        double RE = R;                                   // R^E
#pragma unroll
        for (int s = 1; s < E; s <<= 1) RE *= RE;
        double pw = RE;
#pragma unroll
        for (int off = 1; off < LPM; off <<= 1) {
            const double n = __shfl_up_sync(0xffffffffu, inc, off, LPM);
            if (l >= off) inc = fma(pw, n, inc);
            pw *= pw;
        }
        double run = __shfl_up_sync(0xffffffffu, inc, 1, LPM);
        if (l == 0) run = 0.0;
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const double a = A[e];
            A[e] = run;
            run = fma(R, run, a);
            if (l * E + e < nc) B[e] = fma(K, A[e], B[e]);
        }
        inc = 0.0;
#pragma unroll
        for (int e = E - 1; e >= 0; --e) inc = fma(R, inc, B[e]);
        pw = RE;
#pragma unroll
        for (int off = 1; off < LPM; off <<= 1) {
            const double n = __shfl_down_sync(0xffffffffu, inc, off, LPM);
            if (l + off < LPM) inc = fma(pw, n, inc);
            pw *= pw;
        }
        const double h0 = __shfl_sync(0xffffffffu, inc, 0, LPM) * sC[2 * TX + sm];   // w_0 / (1 − R^{2nc})
        run = __shfl_down_sync(0xffffffffu, inc, 1, LPM);
        if (l == LPM - 1) run = 0.0;
#pragma unroll
        for (int e = E - 1; e >= 0; --e) {               // B[e] ← first w of the next chunk
            const double own_w = B[e];
            B[e] = run;
            run = fma(R, run, own_w);
        }
        const int L = nc / E, lb = l < L ? L - 1 - l : 0;   // lanes in use (E divides nc), distance to the last
        double Rl = 1.0, Rb = 1.0;                       // → R^{lE}, R^{(L−1−l)E}
        pw = RE;
#pragma unroll
        for (int off = 1; off < LPM; off <<= 1) {
            if (l & off) Rl *= pw;
            if (lb & off) Rb *= pw;
            pw *= pw;
        }
        double Rn = __shfl_sync(0xffffffffu, Rb, 0, LPM);   // R^{(L−1)E} → R^{nc}
#pragma unroll
        for (int e = 0; e < E; ++e) Rn *= R;
        const double g0 = -h0 * sC[3 * TX + sm];
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const int cc = l * E + e;
            double dn = Rn * Rb;                         // R^{2nc−cc−1}: from the lane's last chunk down
#pragma unroll
            for (int u = e; u < E - 1; ++u) dn *= R;
            if (cc < nc) {
                sW[sm * LC + cc] = fma(-h0, Rl * R - dn, B[e]);   // first w of chunk cc+1
                sV[sm * LC + cc] = fma(g0, Rl, A[e]);             // carry into chunk cc
            }
            Rl *= R;
        }
    }
    __syncthreads();
    if (!own || col >= n1) return;
    double carry = sV[x * LC + c];
    w = sW[x * LC + c];
#pragma unroll
    for (int i = 0; i < C; ++i) {
        v[i] += carry;
        carry *= r;
    }
    const double kap = sC[TX + x];
#pragma unroll
    for (int i = C - 1; i >= 0; --i) {
        w = fma(r, w, v[i]);
        v[i] = kap * w;
    }
    T* dst = (SRC == YSRC_EDGES ? out : data) + soff;
    int out0 = 0, out1 = g.n2;
    if constexpr (SRC == YSRC_BOTH) {
        out0 = ys.rowbox ? max(0, ys.rowbox[1] - kBoxBelow) : ys.out0;
        out1 = ys.rowbox ? min(g.n2, ys.rowbox[3] + kBoxAbove) : ys.out1;
    }
#pragma unroll
    for (int i = 0; i < C; ++i) {
        const int j = c * C + i - 1;
        if (SRC == YSRC_BOTH ? j >= out0 && j < out1 : j >= 0) dst[o0 + i * P] = (T)v[i];
    }
}

template <class T, int C, int TX, int LPM, int E, int SRC>
cudaError_t launch_ys(const Geom& g, T* data, SlabMap map, int nslabs, const SpecParams& sp, T* out,
                      const YSource& ys, cudaStream_t st) {
    const size_t smem = SRC == YSRC_EDGES || SRC == YSRC_UNIT ? (size_t)g.nx * sizeof(double) : 0;
    const int threads = (TX * (g.ny / C > LPM ? g.ny / C : LPM) + 31) & ~31;
    return launch_k(y_solve_kernel<T, C, TX, LPM, E, SRC>, dim3((g.n1 + TX - 1) / TX, nslabs), dim3(threads), smem,
                    st, data, map, g, sp, out, ys);
}

// Rows per thread and lanes per mode by ny (a multiple of 8 from 32 to 2048).
// 8 rows up to ny = 512: 64-register threads, at most 512 of them.  From 768 on
// 8 rows would need four chunks per scan lane and spill; 16 rows per thread
// take 156 µs for the six solves of a 1024² x 5-level step against 167.
// TX = 8 modes (64-byte rows in FP64): 4 modes are 1-2% slower at 512² and
// 1024², the loads being half as wide.
template <class T, int SRC>
cudaError_t launch_ys_t(const Geom& g, T* data, SlabMap map, int nslabs, const SpecParams& sp, T* out,
                        const YSource& ys, cudaStream_t st) {
    constexpr int TX = 8;
    const int ny = g.ny;
    if (ny % 8 || ny < 32 || ny > 2048 || (ny > 512 && ny % 64)) return cudaErrorInvalidValue;
    if (ny <= 64) return launch_ys<T, 8, TX, 8, 1, SRC>(g, data, map, nslabs, sp, out, ys, st);
    if (ny <= 128) return launch_ys<T, 8, TX, 16, 1, SRC>(g, data, map, nslabs, sp, out, ys, st);
    if (ny <= 256) return launch_ys<T, 8, TX, 32, 1, SRC>(g, data, map, nslabs, sp, out, ys, st);
    if (ny <= 512) {
        if (ny % 16) return cudaErrorInvalidValue;       // two chunks per scan lane
        return launch_ys<T, 8, TX, 32, 2, SRC>(g, data, map, nslabs, sp, out, ys, st);
    }
    if (ny <= 1024) {
        if (ny % 32) return cudaErrorInvalidValue;
        return launch_ys<T, 16, TX, 32, 2, SRC>(g, data, map, nslabs, sp, out, ys, st);
    }
    return launch_ys<T, 16, TX, 32, 4, SRC>(g, data, map, nslabs, sp, out, ys, st);
}

}  // namespace

cudaError_t launch_y_solve(const Geom& g, void* data, SlabMap map, int nslabs, const SpecParams& sp, cudaStream_t st) {
    if (nslabs <= 0) return cudaSuccess;
    if (sp.f32)
        return launch_ys_t<float, YSRC_DATA>(g, static_cast<float*>(data), map, nslabs, sp, nullptr, YSource{}, st);
    return launch_ys_t<double, YSRC_DATA>(g, static_cast<double*>(data), map, nslabs, sp, nullptr, YSource{}, st);
}

cudaError_t launch_y_solve_edges(const Geom& g, void* out, SlabMap map, int nslabs, const SpecParams& sp,
                                 const BtSynth& bs, cudaStream_t st) {
    if (nslabs <= 0) return cudaSuccess;
    YSource ys;
    ys.edges = bs;
    if (sp.f32) return launch_ys_t<float, YSRC_EDGES>(g, nullptr, map, nslabs, sp, static_cast<float*>(out), ys, st);
    return launch_ys_t<double, YSRC_EDGES>(g, nullptr, map, nslabs, sp, static_cast<double*>(out), ys, st);
}

cudaError_t launch_y_solve_both(const Geom& g, double* data, SlabMap map, int nslabs, const SpecParams& sp,
                                const YSource& ys, cudaStream_t st) {
    return launch_ys_t<double, YSRC_BOTH>(g, data, map, nslabs, sp, nullptr, ys, st);
}

cudaError_t launch_y_solve_unit(const Geom& g, double* data, SlabMap map, int nslabs, const SpecParams& sp,
                                const YSource& ys, cudaStream_t st) {
    return launch_ys_t<double, YSRC_UNIT>(g, data, map, nslabs, sp, nullptr, ys, st);
}

}  // namespace ibpm
