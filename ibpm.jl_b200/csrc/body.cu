// Fluid–body coupling of the IBPM step: the regularisation weights of E
// (src/interface-coupling/interface-coupling.jl:6-137), E itself, the
// projection source C'E'F̃b as a deterministic segmented reduction over
// contributions sorted by target, the dense Schur-complement solve and the
// drag/lift reduction (src/timestepping/timestepping.jl:154-163, 204-223,
// 330-354).
#include "ibpm_internal.cuh"

namespace ibpm {

// Yang et al. (2009) smoothed delta function with support ±3 dr, in the
// rounded-coefficient form of interface-coupling.jl:24-61 (result is δ·h).
__device__ double delta_h(double rf, double rb, double dr) {
    const double r = fabs(rf - rb);
    const double r1 = r / dr, r2 = r1 * r1, r3 = r2 * r1, r4 = r3 * r1;
    if (r1 <= 1.0) {
        const double a5 = asin((1.0 / 2.0) * sqrt(3.0) * (2.0 * r1 - 1.0));
        const double a8 = sqrt(1.0 - 12.0 * r2 + 12.0 * r1);
        return 4.166666667e-2 * r4 + (-0.1388888889 + 3.472222222e-2 * a8) * r3 +
               (-7.121664902e-2 - 5.208333333e-2 * a8 + 0.2405626122 * a5) * r2 +
               (-.2405626122 * a5 - 0.3792313933 + 0.1012731481 * a8) * r1 + 8.0187537413e-2 * a5 -
               4.195601852e-2 * a8 + 0.6485698427;
    } else if (r1 <= 2.0) {
        const double a6 = asin((1.0 / 2.0) * sqrt(3.0) * (-3.0 + 2.0 * r1));
        const double a9 = sqrt(-23.0 + 36.0 * r1 - 12.0 * r2);
        return -6.250000000e-2 * r4 + (0.4861111111 - 1.736111111e-2 * a9) * r3 +
               (-1.143175026 + 7.812500000e-2 * a9 - 0.1202813061 * a6) * r2 +
               (0.8751991178 + 0.3608439183 * a6 - 0.1548032407 * a9) * r1 - 0.2806563809 * a6 +
               8.22848104e-3 + 0.1150173611 * a9;
    } else if (r1 <= 3.0) {
        const double a1 = asin((1.0 / 2.0 * (2.0 * r1 - 5.0)) * sqrt(3.0));
        const double a7 = sqrt(-71.0 - 12.0 * r2 + 60.0 * r1);
        return 2.083333333e-2 * r4 + (3.472222222e-3 * a7 - 0.2638888889) * r3 +
               (1.214391675 - 2.604166667e-2 * a7 + 2.405626122e-2 * a1) * r2 +
               (-0.1202813061 * a1 - 2.449273192 + 7.262731481e-2 * a7) * r1 + 0.1523563211 * a1 +
               1.843201677 - 7.306134259e-2 * a7;
    }
    return 0.0;
}

// ∂δh(rf, rb, dr)/∂rb: −sign(rf − rb)/dr times the r1-derivative of the same
// rounded-coefficient pieces (d asin(√3/2 (2r1 − c))/dr1 = √3/√(1 − ¾(2r1 − c)²),
// d √p/dr1 = p'/(2√p)).  At r = 0 the pieces' derivative is ~1e-9 (not exactly
// zero with rounded coefficients); the sign factor makes it 0 there.
__device__ double delta_h_db(double rf, double rb, double dr) {
    const double d = rf - rb;
    const double r1 = fabs(d) / dr, r2 = r1 * r1, r3 = r2 * r1;
    const double s3 = sqrt(3.0);
    double f;
    if (r1 <= 1.0) {
        const double u = 2.0 * r1 - 1.0;
        const double a5 = asin(0.5 * s3 * u), a8 = sqrt(1.0 - 12.0 * r2 + 12.0 * r1);
        const double da5 = s3 / sqrt(1.0 - 0.75 * u * u), da8 = (6.0 - 12.0 * r1) / a8;
        f = 4 * 4.166666667e-2 * r3 + 3 * (-0.1388888889 + 3.472222222e-2 * a8) * r2 + 3.472222222e-2 * da8 * r3 +
            2 * (-7.121664902e-2 - 5.208333333e-2 * a8 + 0.2405626122 * a5) * r1 +
            (-5.208333333e-2 * da8 + 0.2405626122 * da5) * r2 + (-.2405626122 * a5 - 0.3792313933 + 0.1012731481 * a8) +
            (-.2405626122 * da5 + 0.1012731481 * da8) * r1 + 8.0187537413e-2 * da5 - 4.195601852e-2 * da8;
    } else if (r1 <= 2.0) {
        const double u = 2.0 * r1 - 3.0;
        const double a6 = asin(0.5 * s3 * u), a9 = sqrt(-23.0 + 36.0 * r1 - 12.0 * r2);
        const double da6 = s3 / sqrt(1.0 - 0.75 * u * u), da9 = (18.0 - 12.0 * r1) / a9;
        f = -4 * 6.250000000e-2 * r3 + 3 * (0.4861111111 - 1.736111111e-2 * a9) * r2 - 1.736111111e-2 * da9 * r3 +
            2 * (-1.143175026 + 7.812500000e-2 * a9 - 0.1202813061 * a6) * r1 +
            (7.812500000e-2 * da9 - 0.1202813061 * da6) * r2 + (0.8751991178 + 0.3608439183 * a6 - 0.1548032407 * a9) +
            (0.3608439183 * da6 - 0.1548032407 * da9) * r1 - 0.2806563809 * da6 + 0.1150173611 * da9;
    } else if (r1 <= 3.0) {
        const double u = 2.0 * r1 - 5.0;
        const double a1 = asin(0.5 * u * s3), a7 = sqrt(-71.0 - 12.0 * r2 + 60.0 * r1);
        const double da1 = s3 / sqrt(1.0 - 0.75 * u * u), da7 = (30.0 - 12.0 * r1) / a7;
        f = 4 * 2.083333333e-2 * r3 + 3 * (3.472222222e-3 * a7 - 0.2638888889) * r2 + 3.472222222e-3 * da7 * r3 +
            2 * (1.214391675 - 2.604166667e-2 * a7 + 2.405626122e-2 * a1) * r1 +
            (-2.604166667e-2 * da7 + 2.405626122e-2 * da1) * r2 +
            (-0.1202813061 * a1 - 2.449273192 + 7.262731481e-2 * a7) + (-0.1202813061 * da1 + 7.262731481e-2 * da7) * r1 +
            0.1523563211 * da1 - 7.306134259e-2 * da7;
    } else {
        return 0.0;
    }
    const double sg = d > 0.0 ? 1.0 : (d < 0.0 ? -1.0 : 0.0);
    return -sg * f / dr;
}

// Position derivatives of the weights: wd[kk][0][l][m] = ∂w/∂xb_k and
// wd[kk][1][l][m] = ∂w/∂yb_k for the weights of weights_kernel below.
__global__ void dweights_kernel(BodyDev b, double h, double offx, double offy, double* wd) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= b.nf * 169) return;
    const int kk = t / 169, lm = t % 169, l = lm / 13, m = lm % 13;
    const int comp = kk / b.nb, k = kk % b.nb;
    const double xk = b.xb[k], yk = b.xb[b.nb + k];
    const double x = h * (double)((b.bidx[k] - 1) + (l - 6)) - offx + (comp == 1 ? h / 2 : 0.0);
    const double y = h * (double)((b.bidx[b.nb + k] - 1) + (m - 6)) - offy + (comp == 0 ? h / 2 : 0.0);
    wd[(long long)kk * 338 + lm] = delta_h_db(x, xk, h) * delta_h(y, yk, h);
    wd[(long long)kk * 338 + 169 + lm] = delta_h(x, xk, h) * delta_h_db(y, yk, h);
}

cudaError_t launch_dweights(double h, double offx, double offy, const BodyDev& b, double* wd, cudaStream_t st) {
    const int n = b.nf * 169;
    dweights_kernel<<<(n + 255) / 256, 256, 0, st>>>(b, h, offx, offy, wd);
    return cudaGetLastError();
}

// w[kk][l][m], kk = comp·nb + k: weight of flux point (bidx + l − 6, bidx + m − 6)
// for body point k (interface-coupling.jl:89-96).
__global__ void weights_kernel(BodyDev b, double h, double offx, double offy) {
    pdl_wait();
    pdl_trigger();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= b.nf * 169) return;
    const int kk = t / 169, lm = t % 169, l = lm / 13, m = lm % 13;
    const int comp = kk / b.nb, k = kk % b.nb;
    const double xk = b.xb[k], yk = b.xb[b.nb + k];
    const double x = h * (double)((b.bidx[k] - 1) + (l - 6)) - offx;
    const double y = h * (double)((b.bidx[b.nb + k] - 1) + (m - 6)) - offy;
    double w;
    if (comp == 0) w = delta_h(x, xk, h) * delta_h(y + h / 2, yk, h);
    else w = delta_h(x + h / 2, xk, h) * delta_h(y, yk, h);
    b.w[t] = w;
}

cudaError_t launch_weights(const Geom& g, double h, double offx, double offy, const BodyDev& b,
                           cudaStream_t st) {
    const int n = b.nf * 169;
    weights_kernel<<<(n + 255) / 256, 256, 0, st>>>(b, h, offx, offy);
    return cudaGetLastError();
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// E (regT!, interface-coupling.jl:122-133) on (q + q0) with q = C ψ of level 1
// formed in place: one warp per force component and batch member, two ψ values
// per flux of its 13×13 window, so the flux field itself is neither written nor
// read (its curl launch took 7 µs of a 512² step, and 200 MB per 102 columns of
// B on 400×200).  F[bt*F_bstride + kk*F_kstride].
// A moving grid's base flux (MovingFlux, level 1) replaces the uniform q0x, q0y.
// Moving bodies: F −= ub·h, the body-point velocity term of boundary_forces!
// (timestepping.jl:174-186), when ub is set.
// What bounds it is latency: the weights and indices of fixed bodies (FIXED) are
// constants of the handle, so their loads are issued before the dependency wait.
constexpr int kTaps = (169 + 31) / 32;   // window points per lane

template <bool FIXED>
__global__ void __launch_bounds__(256) E_kernel(BodyDev b, Geom g, const double* __restrict__ psi,
                                                long long psi_bstride, int nbatch, double q0x, double q0y, double* F,
                                                long long F_bstride, long long F_kstride, MovingFlux mv,
                                                const double* __restrict__ ub, double hub) {
    if constexpr (!FIXED) {
        pdl_wait();
        pdl_trigger();
    }
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const bool on = warp < b.nf * nbatch;
    const int bt = on ? warp / b.nf : 0, kk = on ? warp % b.nf : 0;
    const int comp = kk / b.nb, k = kk % b.nb;
    const int bx = b.bidx[k], by = b.bidx[b.nb + k];
    const double* w = b.w + (long long)kk * 169;
    double wt[kTaps];
#pragma unroll
    for (int s = 0; s < kTaps; ++s) wt[s] = lane + 32 * s < 169 ? w[lane + 32 * s] : 0.0;
    if constexpr (FIXED) {
        pdl_wait();
        pdl_trigger();
    }
    if (!on) return;
    CurlAt at;
    at.psi = psi + (long long)bt * psi_bstride;
    at.P = g.P; at.nx = g.nx; at.ny = g.ny;
    at.eb.rc = g.mg > 1 ? at.psi + g.S : nullptr;
    at.eb.P = g.P; at.eb.nx = g.nx; at.eb.ny = g.ny;
    const double* mrow = mv.tab ? moving_row(mv) : nullptr;
    double acc = 0.0;
#pragma unroll
    for (int s = 0; s < kTaps; ++s) {
        const int t = lane + 32 * s;
        if (t < 169) {
            const int I = bx + t / 13 - 6, J = by + t % 13 - 6;
            double qv;
            if (comp == 0) qv = at.x(I, J) + (mrow ? moving_q0x(mv, mrow, J, g.ny, mv.h) : q0x);
            else qv = at.y(I, J) + (mrow ? moving_q0y(mv, mrow, I, g.nx, mv.h) : q0y);
            acc += wt[s] * qv;
        }
    }
    acc = warp_sum(acc);
    if (ub) acc = acc - ub[kk] * hub;
    if (lane == 0) F[(long long)bt * F_bstride + (long long)kk * F_kstride] = acc;
}

cudaError_t launch_E(const Geom& g, const BodyDev& b, const double* psi, long long psi_bstride, int nbatch,
                     double q0x, double q0y, double* F, long long F_stride, bool fixed, cudaStream_t st,
                     const MovingFlux& mv, const double* ub, double hub) {
    // F_stride > 0: batch stride with unit component stride; F_stride < 0:
    // component stride |F_stride| with unit batch stride (columns of B).
    const long long bs = F_stride > 0 ? F_stride : 1;
    const long long ks = F_stride > 0 ? 1 : -F_stride;
    const long long warps = (long long)b.nf * nbatch;
    const int blocks = (int)((warps * 32 + 255) / 256);
    return launch_k(fixed ? E_kernel<true> : E_kernel<false>, dim3(blocks), dim3(256), 0, st, b, g, psi, psi_bstride,
                    nbatch, q0x, q0y, F, bs, ks, mv, ub, hub);
}

// y = A x, A row-major n×n (F̃b .= Binv*F̃b, timestepping.jl:160): WPR warps per
// row, partial sums added in a fixed order.  One read of A bounds it (50 MB at
// n = 2512, 7.7 µs); below that, latency, so with CONST (A not rewritten by the
// step: fixed bodies) the thread's first kGemvPre values of A are loaded before
// the dependency wait.
constexpr int kGemvPre = 8;

template <int WPR, bool CONST>
__global__ void __launch_bounds__(256) gemv_kernel(const double* __restrict__ A, const double* __restrict__ x,
                                                   double* y, int n) {
    constexpr int RPB = 8 / WPR, T = 32 * WPR;           // rows per block, threads per row
    __shared__ double part[8];
    if constexpr (!CONST) {
        pdl_wait();
        pdl_trigger();
    }
    const int row = blockIdx.x * RPB + threadIdx.x / T, t = threadIdx.x % T;
    const double* a = A + (long long)(row < n ? row : 0) * n;
    double pre[kGemvPre];
#pragma unroll
    for (int s = 0; s < kGemvPre; ++s) pre[s] = t + s * T < n ? a[t + s * T] : 0.0;
    if constexpr (CONST) {
        pdl_wait();
        pdl_trigger();
    }
    double acc = 0.0;
#pragma unroll
    for (int s = 0; s < kGemvPre; ++s)
        if (t + s * T < n) acc += pre[s] * x[t + s * T];
#pragma unroll 8
    for (int c = t + kGemvPre * T; c < n; c += T) acc += a[c] * x[c];
    acc = warp_sum(acc);
    if constexpr (WPR == 1) {
        if (t == 0 && row < n) y[row] = acc;
    } else {
        if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
        __syncthreads();
        if (t == 0 && row < n) {
            double s = 0.0;
#pragma unroll
            for (int u = 0; u < WPR; ++u) s += part[(threadIdx.x >> 5) + u];
            y[row] = s;
        }
    }
}

// One warp per row up to n = 256 (eight values per lane); four above, where one
// warp left a 25-step chain per lane at n = 804.
cudaError_t launch_gemv(const double* A, const double* x, double* y, int n, bool constant, cudaStream_t st) {
    if (n <= 256)
        return launch_k(constant ? gemv_kernel<1, true> : gemv_kernel<1, false>, dim3((n + 7) / 8), dim3(256), 0, st, A,
                        x, y, n);
    return launch_k(constant ? gemv_kernel<4, true> : gemv_kernel<4, false>, dim3((n + 1) / 2), dim3(256), 0, st, A, x,
                    y, n);
}

// update_stress! (timestepping.jl:330-354): fb = F̃b (h/dt) ./ ds,
// CD_j = 2 Σ ds fb_x, CL_j = 2 Σ ds fb_y, written to hist[step][2][nbodies]
// for step < hist_cap (a later step writes nothing and sets bit 3 of *status).
// One block; a non-finite CD/CL sets bit 0 of *status.
__device__ __forceinline__ void stress_block(const BodyDev& b, const double* __restrict__ Fb, double h, double dt,
                                             double* hist, int hist_cap, int* counter, int* status) {
    __shared__ double red[2][8];
    const int step = *counter;
    const bool keep = step >= 0 && step < hist_cap;
    if (!keep && threadIdx.x == 0) atomicOr(status, 8);
    const double hdt = h / dt;
    for (int j = 0; j < b.nbodies; ++j) {
        const int p0 = b.body_start[j], p1 = b.body_start[j + 1];
        double sx = 0.0, sy = 0.0;
        for (int p = p0 + threadIdx.x; p < p1; p += blockDim.x) {
            const double ds = b.ds[p];
            sx += ds * ((Fb[p] * hdt) / ds);
            sy += ds * ((Fb[b.nb + p] * hdt) / ds);
        }
        sx = warp_sum(sx);
        sy = warp_sum(sy);
        if ((threadIdx.x & 31) == 0) {
            red[0][threadIdx.x >> 5] = sx;
            red[1][threadIdx.x >> 5] = sy;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            double cd = 0.0, cl = 0.0;
            for (int u = 0; u < 8; ++u) {
                cd += red[0][u];
                cl += red[1][u];
            }
            cd *= 2.0;
            cl *= 2.0;
            if (keep) {
                hist[((long long)step * 2 + 0) * b.nbodies + j] = cd;
                hist[((long long)step * 2 + 1) * b.nbodies + j] = cl;
            }
            if (!isfinite(cd) || !isfinite(cl)) atomicOr(status, 1);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) *counter = step + 1;
}

__global__ void stress_kernel(BodyDev b, const double* __restrict__ Fb, double h, double dt, double* hist,
                              int hist_cap, int* counter, int* status) {
    pdl_wait();
    pdl_trigger();
    stress_block(b, Fb, h, dt, hist, hist_cap, counter, status);
}

cudaError_t launch_stress(const BodyDev& b, const double* Fb, double h, double dt, double* hist, int hist_cap,
                          int* counter, int* status, cudaStream_t st) {
    return launch_k(stress_kernel, dim3(1), dim3(256), 0, st, b, Fb, h, dt, hist, hist_cap, counter, status);
}

// update_stress! and the projection source in one launch (both read only F̃b):
// block 0 reduces CD/CL (and advances the step counter), the other blocks form
// Γsrc = C'(E' F̃b) at the Γ points whose rot! stencil touches a regularised
// flux point (timestepping.jl:217, curl.jl:22-34): Γ = (qx₁ − qx₂) +
// (qy₁ − qy₂) over the point's four fluxes, each flux the sum over its sorted
// contributor list (interface-coupling.jl:103-107).  One warp per Γ point:
// the lanes take the contributors of all four fluxes (about 50 at one point
// per h), with the signs of rot!, and a shuffle tree adds them in a fixed
// order, so the result is deterministic (the reference adds sequentially;
// the two agree to round-off).  The lists and weights of fixed bodies are
// constants: a lane's first contributor of each flux (lists of up to 32) is
// looked up before the dependency wait, three dependent loads off the chain.
__global__ void __launch_bounds__(256) stress_src_kernel(BodyDev b, const double* __restrict__ Fb, double h, double dt,
                                                         double* hist, int hist_cap, int* counter, int* status,
                                                         double* Gsrc) {
    if (blockIdx.x == 0) {
        pdl_wait();
        pdl_trigger();
        stress_block(b, Fb, h, dt, hist, hist_cap, counter, status);
        return;
    }
    const int p = ((blockIdx.x - 1) * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    const bool on = p < b.n_src;
    int next[4], end[4], kf[4];
    double wf[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int row = on ? b.src_rows[4 * p + r] : -1;
        next[r] = row < 0 ? 0 : b.et_ptr[row] + lane;
        end[r] = row < 0 ? 0 : b.et_ptr[row + 1];
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const bool any = next[r] < end[r];
        kf[r] = any ? b.et_k[next[r]] : 0;
        wf[r] = any ? b.w[b.et_w[next[r]]] : 0.0;
    }
    pdl_wait();
    pdl_trigger();
    if (!on) return;
    double v = 0.0;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        double acc = wf[r] * Fb[kf[r]];
        for (int e = next[r] + 32; e < end[r]; e += 32) acc += b.w[b.et_w[e]] * Fb[b.et_k[e]];
        v += (r == 0 || r == 2) ? acc : -acc;
    }
    v = warp_sum(v);
    if (lane == 0) Gsrc[b.src_pts[p]] = v;
}

cudaError_t launch_stress_src(const BodyDev& b, const double* Fb, double h, double dt, double* hist, int hist_cap,
                              int* counter, int* status, double* Gsrc, cudaStream_t st) {
    const long long threads = (long long)b.n_src * 32;
    const unsigned blocks = 1 + (unsigned)((threads + 255) / 256);
    return launch_k(stress_src_kernel, dim3(blocks), dim3(256), 0, st, b, Fb, h, dt, hist, hist_cap, counter, status,
                    Gsrc);
}

// ---------------------------------------------------------------------------
// Bodies moved by a MotionFunction (move_body!, move-body-utils.jl:86-133):
// point p of body j at the step's row r = (x, y, cos θ, sin θ, ẋ, ẏ, θ̇) of the
// motion table is xb = (x, y) + Rx x0, ub = (ẋ, ẏ) + Ru x0 with
// Rx = [c −s; s c], Ru = θ̇ [−s −c; c −s], evaluated in the reference's order
// without fused multiply-adds; body_idx = floor((xb + off)/h)
// (interface-coupling.jl:86-87).  A point whose 13×13 window would leave the
// finest grid sets bit 4 of the status word and is clamped inside, so that no
// later kernel reads outside the grid.  The bounding box of the windows'
// centres (min/max body_idx) is accumulated for the projection source.
// ---------------------------------------------------------------------------
__global__ void kinematics_kernel(BodyDev b, Geom g, const double* __restrict__ x0, const double* __restrict__ tab,
                                  const int* __restrict__ step, double h, double offx, double offy, double* xb,
                                  int* bidx, double* ub, int* bbox, int* status) {
    pdl_wait();
    pdl_trigger();
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= b.nb) return;
    int j = 0;
    while (j + 1 < b.nbodies && p >= b.body_start[j + 1]) ++j;
    const double* r = tab + ((long long)(*step) * b.nbodies + j) * 8;
    const double X = x0[p], Y = x0[b.nb + p];
    const double c = r[2], s = r[3], thd = r[6];
    const double xp = __dadd_rn(r[0], __dadd_rn(__dmul_rn(c, X), __dmul_rn(-s, Y)));
    const double yp = __dadd_rn(r[1], __dadd_rn(__dmul_rn(s, X), __dmul_rn(c, Y)));
    xb[p] = xp;
    xb[b.nb + p] = yp;
    ub[p] = __dadd_rn(r[4], __dadd_rn(__dmul_rn(__dmul_rn(thd, -s), X), __dmul_rn(__dmul_rn(thd, -c), Y)));
    ub[b.nb + p] = __dadd_rn(r[5], __dadd_rn(__dmul_rn(__dmul_rn(thd, c), X), __dmul_rn(__dmul_rn(thd, -s), Y)));
    double fx = floor((xp + offx) / h), fy = floor((yp + offy) / h);
    if (!window_inside(g, fx, fy)) {
        atomicOr(status, 4);
        fx = fmin(fmax(fx, 7.0), g.nx - 6.0);            // fmax of no number is 7
        fy = fmin(fmax(fy, 7.0), g.ny - 6.0);
    }
    const int bx = (int)fx, by = (int)fy;
    bidx[p] = bx;
    bidx[b.nb + p] = by;
    atomicMin(&bbox[0], bx);
    atomicMin(&bbox[1], by);
    atomicMax(&bbox[2], bx);
    atomicMax(&bbox[3], by);
}

cudaError_t launch_kinematics(const Geom& g, const BodyDev& b, const double* x0, const double* tab, const int* step,
                              double h, double offx, double offy, double* xb, int* bidx, double* ub, int* bbox,
                              int* status, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(bbox, 0x7f, 2 * sizeof(int), st);   // min slots: a large positive int
    if (e == cudaSuccess) e = cudaMemsetAsync(bbox + 2, 0x80, 2 * sizeof(int), st);  // max slots: a large negative one
    if (e != cudaSuccess) return e;
    return launch_k(kinematics_kernel, dim3((b.nb + 127) / 128), dim3(128), 0, st, b, g, x0, tab, step, h, offx, offy,
                    xb, bidx, ub, bbox, status);
}

// C'E'F̃b on the level-1 slab for moving bodies, every Γ point in gather form:
// each regularised flux sums w·F̃b over the body points whose window holds it,
// in ascending point order (reg!, interface-coupling.jl:99-119), then
// Γ[i-1, j-1] = (qx[i, j-1] − qx[i, j]) + (qy[i, j] − qy[i-1, j]) (rot!).
// Points outside the windows' bounding box are written 0.
__global__ void proj_src_moving_kernel(BodyDev b, Geom g, const double* __restrict__ Fb, const int* __restrict__ bbox,
                                       double* Gsrc) {
    pdl_wait();
    pdl_trigger();
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)g.n1 * g.n2) return;
    const int i0 = (int)(t % g.n1), j0 = (int)(t / g.n1);
    const int i = i0 + 2, j = j0 + 2;  // Julia indices of the fluxes around Γ[i0+1, j0+1]
    double v = 0.0;
    if (i + 1 >= bbox[0] - 6 && i - 1 <= bbox[2] + 6 && j + 1 >= bbox[1] - 6 && j - 1 <= bbox[3] + 6) {
        auto flux = [&](int comp, int I, int J) -> double {
            double q = 0.0;
            for (int k = 0; k < b.nb; ++k) {
                const int l = I - b.bidx[k] + 6, m = J - b.bidx[b.nb + k] + 6;
                if (l >= 0 && l < 13 && m >= 0 && m < 13) {
                    const int kk = comp * b.nb + k;
                    q = __dadd_rn(q, __dmul_rn(b.w[(long long)kk * 169 + l * 13 + m], Fb[kk]));
                }
            }
            return q;
        };
        v = (flux(0, i, j - 1) - flux(0, i, j)) + (flux(1, i, j) - flux(1, i - 1, j));
    }
    Gsrc[(long long)j0 * g.P + i0] = v;
}

cudaError_t launch_proj_src_moving(const Geom& g, const BodyDev& b, const double* Fb, const int* bbox, double* Gsrc,
                                   cudaStream_t st) {
    const long long n = (long long)g.n1 * g.n2;
    return launch_k(proj_src_moving_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, st, b, g, Fb, bbox, Gsrc);
}

__global__ void info_to_status_kernel(const int* info, int* status) {
    if (*info) atomicOr(status, 2);
}

cudaError_t launch_info_to_status(const int* info, int* status, cudaStream_t st) {
    info_to_status_kernel<<<1, 1, 0, st>>>(info, status);
    return cudaGetLastError();
}

}  // namespace ibpm
