// Grid stencils of the IBPM step: the right-hand side of the trial solve
// (nonlinear term + AB2 + explicit viscous term + cross-level BCs), coarsify!
// and the multigrid curl.  Index comments use the reference's 1-based
// (Julia) indices; device arrays are 0-based (see ibpm_internal.cuh).
#include "ibpm_internal.cuh"

namespace ibpm {

// ---------------------------------------------------------------------------
// Trial right-hand side, one thread per Γ point of one level:
//   bc   = get_bc!(Γ[lev+1])                   (timestepping.jl:101-106)
//   rhsbc= apply_bc!(0, bc, 0.25 dt/(Re hc²))
//   N    = nonlinear!(Γ, q, q0, 0.25 bc)       (nonlinear.jl:168-201)
//   rhs  = A Γ + β1 dt N + β2 dt Nprev + rhsbc  (timestepping.jl:111-118)
// A Γ is evaluated as the 5-point stencil Γ + c (Σ neighbours − 4Γ), c =
// dt/(2 Re hc²), with zero Dirichlet edges: the operator the reference applies
// through two DSTs with the eigenvalues 1 − Λ c (laplacian.jl:73-76), whose
// eigenvectors are exactly the DST-I basis.
// ---------------------------------------------------------------------------
// In N = C' fq the product at the point's own vertex enters both x-faces (and
// both y-faces) with opposite signs, so only the four neighbours are left:
//   4 hc² N = Qy(i+1, j) Γ(i, j−1) − Qy(i+1, j+2) Γ(i, j+1)
//           + Qx(i, j+1) Γ(i−1, j) − Qx(i+2, j+1) Γ(i+1, j),
// 13 loads per point with the stencil's, where forming the four products of fq
// read about 30 values and tested for the edges at each (five levels of 511²
// 31 -> 22 µs, of 1023² 108 -> 73 µs, timed by events in the step; the bytes of
// the latter, 252 MB, take 39 µs).  Bound by L1 and L2 requests.
// LIN: the linearised problem's term (nonlinear.jl:45-65, 144-163),
//   N = C'(DP(Q, ΓB) + DP(QB, Γ)) / (4 hc²),
// Q the face sums of q without base flux, QB those of the base state with its
// base flux, both products using this state's edge values ¼ get_bc!(Γ[l+1])
// (the reference passes the perturbation's Γbc to the ΓB product too).
// MOV: a moving grid's per-face base flux (MovingFlux) instead of q0x, q0y.
// GRP: the simulations of a batch group, blockIdx.z = simulation · mg + level,
// each with its own arguments in ga[simulation] (its fields, coefficients).
template <bool LIN, bool MOV>
__device__ __forceinline__ void trial_point(const RhsArgs& a, const Geom& g, int lev, int i0, int j0) {
    const int nx = g.nx, ny = g.ny, n1 = g.n1, n2 = g.n2, P = g.P;
    const double* G = a.G + a.Gmap.off(lev);
    const double* q = a.q + (long long)lev * g.nq;
    const int o = j0 * P + i0;                           // a level is below 2^31 values
    const int ox = j0 * (nx + 1) + i0;                   // 0-based flux (i0, j0) of the x-faces
    const int oy = j0 * nx + i0;                         // … of the y-faces

    // Γ at the point and its four neighbours: the edge values ¼ get_bc! beyond
    // the level's edges for the products (gs …), zero for the viscous term (zs …)
    const double gc = G[o];
    double gw, ge, gs, gn, zw, ze, zs, zn, rbc = 0.0;
    if (i0 > 0 && i0 < n1 - 1 && j0 > 0 && j0 < n2 - 1) {
        zw = gw = G[o - 1];
        ze = ge = G[o + 1];
        zs = gs = G[o - P];
        zn = gn = G[o + P];
    } else {
        CoarseBC cb;
        cb.rc = (lev < a.mg - 1) ? a.G + a.Gmap.off(lev + 1) : nullptr;
        cb.P = P; cb.nx = nx; cb.ny = ny;
        // apply_bc!(rhsbc = 0, bc, fac) (mg-utils.jl:43-60), in the order bottom, top, left, right
        const double fac = a.fac_bc[lev];
        zs = zn = zw = ze = 0.0;
        if (j0 == 0) { const double b = cb.bot(i0 + 1); gs = 0.25 * b; rbc += fac * b; }
        else zs = gs = G[o - P];
        if (j0 == n2 - 1) { const double b = cb.top(i0 + 1); gn = 0.25 * b; rbc += fac * b; }
        else zn = gn = G[o + P];
        if (i0 == 0) { const double b = cb.left(j0 + 1); gw = 0.25 * b; rbc += fac * b; }
        else zw = gw = G[o - 1];
        if (i0 == n1 - 1) { const double b = cb.right(j0 + 1); ge = 0.25 * b; rbc += fac * b; }
        else ze = ge = G[o + 1];
    }
    // face sums of avg_flux (nonlinear.jl:17-38) at the four faces, without
    // base flux: Qx of rows j, j+1 at x-faces I = i, i+2; Qy of columns i, i+1
    // at y-faces J = j, j+2 (1-based; 0-based offsets below)
    struct Faces { double w, e, s, n; };
    auto faces = [&](const double* f) -> Faces {
        const double* fy = f + g.nu;
        return {f[ox + nx + 1] + f[ox], f[ox + 2 + nx + 1] + f[ox + 2], fy[oy + 1] + fy[oy],
                fy[oy + 2 * nx + 1] + fy[oy + 2 * nx]};
    };
    Faces Q = faces(q);
    double N;
    if constexpr (!LIN) {
        if constexpr (MOV) {
            // the base flux varies along y on x-faces and along x on y-faces
            const double* mrow = moving_row(a.mv);
            const double hc = ldexp(a.mv.h, lev);
            const double bx = moving_q0x(a.mv, mrow, j0 + 2, ny, hc) + moving_q0x(a.mv, mrow, j0 + 1, ny, hc);
            const double by = moving_q0y(a.mv, mrow, i0 + 2, nx, hc) + moving_q0y(a.mv, mrow, i0 + 1, nx, hc);
            Q.w += bx; Q.e += bx; Q.s += by; Q.n += by;
        } else {
            const double bx = 2.0 * a.q0x[lev], by = 2.0 * a.q0y[lev];
            Q.w += bx; Q.e += bx; Q.s += by; Q.n += by;
        }
        N = ((Q.s * gs - Q.n * gn) + (Q.w * gw - Q.e * ge)) * a.nl_scale[lev];
    } else {
        const double* GB = a.GB + a.Gmap.off(lev);       // base Γ, this state's edge values
        const double bw = i0 > 0 ? GB[o - 1] : gw, be = i0 < n1 - 1 ? GB[o + 1] : ge;
        const double bs = j0 > 0 ? GB[o - P] : gs, bn = j0 < n2 - 1 ? GB[o + P] : gn;
        Faces QB = faces(a.qB + (long long)lev * g.nq);
        const double bx = 2.0 * a.q0Bx[lev], by = 2.0 * a.q0By[lev];
        QB.w += bx; QB.e += bx; QB.s += by; QB.n += by;
        N = (((Q.s * bs + QB.s * gs) - (Q.n * bn + QB.n * gn)) + ((Q.w * bw + QB.w * gw) - (Q.e * be + QB.e * ge))) *
            a.nl_scale[lev];
    }
    // explicit viscous operator
    const double AG = gc + a.c_lap[lev] * ((((ze + zw) + zn) + zs) - 4.0 * gc);
    const long long oo = a.Gmap.off(lev) + o;
    const double Np = a.Nprev[oo];
    a.Nnew[oo] = N;
    a.rhs[oo] = ((AG + a.b1dt * N) + a.b2dt * Np) + rbc;
}

template <bool LIN, bool MOV, bool GRP = false>
__global__ void __launch_bounds__(256) trial_rhs_kernel(const __grid_constant__ RhsArgs a0,
                                                        const RhsArgs* __restrict__ ga, Geom g) {
    pdl_wait();
    pdl_trigger();
    const RhsArgs& a = GRP ? ga[blockIdx.z / g.mg] : a0;
    const int i0 = blockIdx.x * blockDim.x + threadIdx.x;
    const int j0 = blockIdx.y * blockDim.y + threadIdx.y;
    const int lev = GRP ? (int)(blockIdx.z % g.mg) : (int)blockIdx.z;
    if (i0 >= g.n1 || j0 >= g.n2) return;
    trial_point<LIN, MOV>(a, g, lev, i0, j0);
}

// The same for 2 × 2 points per thread (fixed grid, not linearised): 40 values read
// for 4 points instead of 56, most in aligned pairs, so 30 load instructions instead
// of 56.  Points on the rim, the columns 0, 1, n1 − 1 and the rows 0, 1, n2 − 1, are
// the business of extra blocks, one point per thread, so that no warp takes both
// paths (inside the tiles' blocks they cost 4 µs of a step at any size).  1023² x 5
// levels: 65 -> 43 µs, of which the bytes take 39; 511² x 5 22 -> 14.
template <bool GRP>
__global__ void __launch_bounds__(256) trial_rhs_tile_kernel(const __grid_constant__ RhsArgs a0,
                                                             const RhsArgs* __restrict__ ga, Geom g) {
    pdl_wait();
    pdl_trigger();
    const RhsArgs& a = GRP ? ga[blockIdx.z / g.mg] : a0;
    const int lev = GRP ? (int)(blockIdx.z % g.mg) : (int)blockIdx.z;
    const int nx = g.nx, n1 = g.n1, n2 = g.n2, P = g.P;
    const int rim0 = (n2 + 15) / 16;                     // the blocks of tiles are rows 0 … rim0 − 1
    if ((int)blockIdx.y >= rim0) {
        // the columns 0, 1, n1 − 1, then what is left of the rows 0, 1, n2 − 1
        const int t = ((blockIdx.y - rim0) * gridDim.x + blockIdx.x) * 256 + threadIdx.y * 32 + threadIdx.x;
        const int u = t - 3 * n2;
        if (u >= 3 * (n1 - 3)) return;
        const int s = t < 3 * n2 ? t / n2 : u / (n1 - 3);
        const int i = t < 3 * n2 ? (s < 2 ? s : n1 - 1) : 2 + u - s * (n1 - 3);
        const int j = t < 3 * n2 ? t - s * n2 : (s < 2 ? s : n2 - 1);
        trial_point<false, false>(a, g, lev, i, j);
        return;
    }
    const int i0 = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
    const int j0 = 2 * (blockIdx.y * blockDim.y + threadIdx.y);
    if (i0 == 0 || i0 >= n1 - 1 || j0 == 0 || j0 >= n2 - 1) return;
    // i0, P, nx, the level's and the y-faces' offsets are even: pairs are aligned
    auto two = [](const double* p) { return *reinterpret_cast<const double2*>(p); };
    const long long oo = a.Gmap.off(lev) + j0 * P + i0;
    const double* G = a.G + oo;
    const double* fx = a.q + (long long)lev * g.nq + j0 * (nx + 1) + i0;
    const double* fy = a.q + (long long)lev * g.nq + g.nu + j0 * nx + i0;
    double2 c[4], y2[4], Np[2];
    double w[2], e[2], x[3][4], y1[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        c[r] = two(G + (r - 1) * P);
        y2[r] = two(fy + r * nx);
        y1[r] = fy[r * nx + 2];
    }
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int k = 0; k < 4; ++k) x[r][k] = fx[r * (nx + 1) + k];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        w[r] = G[r * P - 1];
        e[r] = G[r * P + 2];
        Np[r] = two(a.Nprev + oo + r * P);
    }
    const double bx = 2.0 * a.q0x[lev], by = 2.0 * a.q0y[lev], sc = a.nl_scale[lev], cl = a.c_lap[lev];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        double N[2], R[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const double gc = k ? c[r + 1].y : c[r + 1].x, gs = k ? c[r].y : c[r].x, gn = k ? c[r + 2].y : c[r + 2].x;
            const double gw = k ? c[r + 1].x : w[r], ge = k ? e[r] : c[r + 1].y;
            const double Qw = (x[r + 1][k] + x[r][k]) + bx, Qe = (x[r + 1][k + 2] + x[r][k + 2]) + bx;
            const double Qs = (k ? y1[r] + y2[r].y : y2[r].y + y2[r].x) + by;
            const double Qn = (k ? y1[r + 2] + y2[r + 2].y : y2[r + 2].y + y2[r + 2].x) + by;
            N[k] = ((Qs * gs - Qn * gn) + (Qw * gw - Qe * ge)) * sc;
            const double AG = gc + cl * ((((ge + gw) + gn) + gs) - 4.0 * gc);
            R[k] = (AG + a.b1dt * N[k]) + a.b2dt * (k ? Np[r].y : Np[r].x);
        }
        *reinterpret_cast<double2*>(a.Nnew + oo + r * P) = make_double2(N[0], N[1]);
        *reinterpret_cast<double2*>(a.rhs + oo + r * P) = make_double2(R[0], R[1]);
    }
}

// From 2^19 points of a simulation on, the tiles are the faster (512² x 3 levels
// 137.5 -> 136.6 µs per step, x 5 177.2 -> 174.0, 1024² x 3 326 -> 313, x 5 491 ->
// 471); below, the step loses up to 1 µs to them (64² x 3 60.5 -> 61.5, 256² x 4
// 100.3 -> 101.2, 400x200 x 5 even): too few threads, each with a longer chain.
// The size of one simulation decides, also in a group: a member's results do not
// depend on its group.
static bool trial_tiled(const Geom& g) { return (long long)g.n1 * g.n2 * g.mg >= 1 << 19; }
static dim3 trial_tiles(const Geom& g, int nsim) {
    const int bx = (g.n1 + 63) / 64, rim = (3 * g.n2 + 3 * (g.n1 - 3) + 255) / 256;
    return dim3(bx, (g.n2 + 15) / 16 + (rim + bx - 1) / bx, nsim * g.mg);
}

cudaError_t launch_trial_rhs(const Geom& g, const RhsArgs& a, cudaStream_t st) {
    dim3 blk(32, 8);
    dim3 grid((g.n1 + 31) / 32, (g.n2 + 7) / 8, a.mg);
    const RhsArgs* none = nullptr;
    if (a.GB) return launch_k(trial_rhs_kernel<true, false>, grid, blk, 0, st, a, none, g);
    if (a.mv.tab) return launch_k(trial_rhs_kernel<false, true>, grid, blk, 0, st, a, none, g);
    if (trial_tiled(g)) return launch_k(trial_rhs_tile_kernel<false>, trial_tiles(g, 1), blk, 0, st, a, none, g);
    return launch_k(trial_rhs_kernel<false, false>, grid, blk, 0, st, a, none, g);
}

cudaError_t launch_trial_rhs_group(const Geom& g, const RhsArgs& a0, const RhsArgs* ga, int nsim, cudaStream_t st) {
    dim3 blk(32, 8);
    if (trial_tiled(g)) return launch_k(trial_rhs_tile_kernel<true>, trial_tiles(g, nsim), blk, 0, st, a0, ga, g);
    dim3 grid((g.n1 + 31) / 32, (g.n2 + 7) / 8, nsim * g.mg);
    return launch_k(trial_rhs_kernel<false, false, true>, grid, blk, 0, st, a0, ga, g);
}

// ---------------------------------------------------------------------------
// coarsify! (mg-utils.jl:71-106): the centre half of the coarse level gets the
// full-weighting restriction of the fine level, Γc[ic, jc] =
//   Γ[i,j] + ½ (Γ[i+1,j] + Γ[i,j+1] + Γ[i-1,j] + Γ[i,j-1])
//          + ¼ (Γ[i+1,j+1] + Γ[i+1,j-1] + Γ[i-1,j-1] + Γ[i-1,j+1]),
// i = 2:2:nx-2 ↔ ic = nx/4 + i/2.
// ---------------------------------------------------------------------------
__global__ void coarsify_kernel(double* G, SlabMap fmap, SlabMap cmap, Geom g) {
    pdl_wait();
    pdl_trigger();
    const int nxc = g.nx / 2 - 1, nyc = g.ny / 2 - 1;
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    const int b = blockIdx.y * blockDim.y + threadIdx.y;
    if (a >= nxc || b >= nyc) return;
    const int P = g.P;
    const double* F = G + fmap.off(blockIdx.z);
    double* C = G + cmap.off(blockIdx.z);
    const int i = 2 * a + 1, j = 2 * b + 1;  // 0-based fine point
    auto f = [&](int ii, int jj) -> double { return F[(long long)jj * P + ii]; };
    const double e = ((f(i + 1, j) + f(i, j + 1)) + f(i - 1, j)) + f(i, j - 1);
    const double d = ((f(i + 1, j + 1) + f(i + 1, j - 1)) + f(i - 1, j - 1)) + f(i - 1, j + 1);
    C[(long long)(g.ny / 4 + b) * P + (g.nx / 4 + a)] = (f(i, j) + 0.5 * e) + 0.25 * d;
}

cudaError_t launch_coarsify(const Geom& g, double* G, SlabMap fine_map, SlabMap coarse_map, int nslabs,
                            cudaStream_t st) {
    dim3 blk(32, 8);
    dim3 grid((g.nx / 2 - 1 + 31) / 32, (g.ny / 2 - 1 + 7) / 8, nslabs);
    return launch_k(coarsify_kernel, grid, blk, 0, st, G, fine_map, coarse_map, g);
}

// ---------------------------------------------------------------------------
// Multigrid curl (curl.jl:81-116): q = C ψ with edge streamfunction from
// ψbc = get_bc!(ψ[lev+1]) (zero on the coarsest level).  Reproduces the
// reference exactly, including the bottom row of x-fluxes reading ψbc[(B-1)+i]
// (curl.jl:92), i.e. edge vertex i-2, where the top row reads vertex i-1.
// Each thread takes column I of kCurlRows rows and writes both fluxes, so a value
// of ψ is loaded about twice instead of four times and the indices need no
// division (one thread per flux element did both): per step of 512² x 5 levels
// 34 -> 22 µs, of 1024² x 5 95 -> 41 µs (events; the latter moves 150 MB, 23 µs).
// blockIdx.z = batch × levels.
// ---------------------------------------------------------------------------
constexpr int kCurlRows = 4;

__global__ void __launch_bounds__(256) curl_kernel(CurlArgs a, Geom g) {
    pdl_wait();
    pdl_trigger();
    const int I = blockIdx.x * blockDim.x + threadIdx.x + 1;                    // 1 … nx + 1
    const int J0 = (blockIdx.y * blockDim.y + threadIdx.y) * kCurlRows + 1;     // rows J0 … of 1 … ny + 1
    const int z = blockIdx.z;
    const int lev = a.psi_map.level(z);
    const int nx = g.nx, ny = g.ny, P = g.P;
    if (I > nx + 1 || J0 > ny + 1) return;
    const double* psi = a.psi + a.psi_map.off(z);
    double* qx = a.q + (long long)a.psi_map.batch(z) * a.q_bstride + (long long)(lev - a.q_lev0) * a.q_lstride;
    double* qy = qx + g.nu;
    if (I > 1 && I < nx && J0 > 1 && J0 + kCurlRows <= ny) {
        const double* p = psi + (J0 - 2) * P + (I - 2);  // ψ(I−1, J0−1)
        double w[kCurlRows + 1], e[kCurlRows];
#pragma unroll
        for (int r = 0; r <= kCurlRows; ++r) w[r] = p[r * P];
#pragma unroll
        for (int r = 0; r < kCurlRows; ++r) e[r] = p[r * P + 1];
        const int ox = (I - 1) + (J0 - 1) * (nx + 1), oy = (I - 1) + (J0 - 1) * nx;
#pragma unroll
        for (int r = 0; r < kCurlRows; ++r) {
            qx[ox + r * (nx + 1)] = w[r + 1] - w[r];
            qy[oy + r * nx] = w[r] - e[r];
        }
        return;
    }
    CurlAt at;
    at.psi = psi; at.P = P; at.nx = nx; at.ny = ny;
    at.eb.rc = (lev < a.mg - 1) ? a.coarse + a.coarse_map.off(z) : nullptr;
    at.eb.P = P; at.eb.nx = nx; at.eb.ny = ny;
    for (int r = 0; r < kCurlRows; ++r) {
        const int J = J0 + r;
        if (J <= ny) qx[(I - 1) + (J - 1) * (nx + 1)] = at.x(I, J);
        if (J <= ny + 1 && I <= nx) qy[(I - 1) + (J - 1) * nx] = at.y(I, J);
    }
}

cudaError_t launch_curl(const Geom& g, const CurlArgs& a, cudaStream_t st) {
    dim3 blk(32, 8);
    dim3 grid((g.nx + 1 + 31) / 32, (g.ny + 1 + 8 * kCurlRows - 1) / (8 * kCurlRows), a.nlev * a.nbatch);
    return launch_k(curl_kernel, grid, blk, 0, st, a, g);
}

// ---------------------------------------------------------------------------
// FP64 residual of one refinement sweep of vort2flux! on every level at once,
// stored in FP32 (it is small: the change of ψ since its previous solve):
//     r_ℓ = Γ_ℓ + apply_bc!(get_bc!(ψ_{ℓ+1})) − L ψ_ℓ
// with L x = 4x − Σ neighbours (zero Dirichlet edges), the operator the
// DST-I solve with Λ inverts (laplacian.jl:14-41), and the edge term of a
// level of vort2flux! (curl.jl:151-158, mg-utils.jl:7-60); none at the
// coarsest level.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) resid_lap_kernel(const double* __restrict__ G, const double* __restrict__ psi,
                                                        float* r, Geom g) {
    pdl_wait();
    pdl_trigger();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    // slab z = simulation · mg + level (simulations mg slabs apart)
    const int z = blockIdx.z, lev = z % g.mg;
    const int n1 = g.n1, n2 = g.n2, P = g.P;
    if (i >= n1 || j >= n2) return;
    const double* x = psi + (long long)z * g.S;
    const long long o = (long long)j * P + i;
    const double xc = x[o];
    double nb = 0.0;
    if (i > 0) nb += x[o - 1];
    if (i + 1 < n1) nb += x[o + 1];
    if (j > 0) nb += x[o - P];
    if (j + 1 < n2) nb += x[o + P];
    double v = G[(long long)z * g.S + o];
    if (lev + 1 < g.mg) {
        CoarseBC cb;
        cb.rc = psi + (long long)(z + 1) * g.S; cb.P = P; cb.nx = g.nx; cb.ny = g.ny;
        if (j == 0) v += cb.bot(i + 1);
        if (j == n2 - 1) v += cb.top(i + 1);
        if (i == 0) v += cb.left(j + 1);
        if (i == n1 - 1) v += cb.right(j + 1);
    }
    v -= 4.0 * xc - nb;
    r[(long long)z * g.S + o] = (float)v;
}

cudaError_t launch_resid_lap(const Geom& g, const double* G, const double* psi, float* r, int nsim, cudaStream_t st) {
    dim3 blk(32, 8);
    dim3 grid((g.n1 + 31) / 32, (g.n2 + 7) / 8, g.mg * nsim);
    return launch_k(resid_lap_kernel, grid, blk, 0, st, G, psi, r, g);
}

}  // namespace ibpm
