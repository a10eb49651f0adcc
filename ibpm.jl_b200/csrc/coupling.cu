// The lists of the regularisation E' = C-ordered sums over force components
// (reg!, interface-coupling.jl:99-119) and of the projection source C'E', built
// on the device when a problem is made: E' as CSR over the touched flux points in
// ascending flux index, each point's contributors in ascending component order,
// and the Γ points whose rot! stencil touches one of them, in ascending order.
//
// A count per flux point, one scan over the fluxes and one over the Γ points give
// every list its place; the contributors are scattered in any order and then
// ranked by component inside their row, so the lists do not depend on the order
// of the atomics.  Bound by the launches at the usual sizes (8 kernels over 80 000
// to 520 000 fluxes and some 50 000 contributors); a problem of 200² with 314 force
// components is made in 6.4 ms, with a sorted map on the host it took 12.6 (of
// which 6 in the map).
#include "ibpm_internal.cuh"

namespace ibpm {

namespace {

constexpr int kScanThreads = 256, kScanItems = 8, kScanBlock = kScanThreads * kScanItems;

// Flux of contributor (kk, t): component kk's window point t = l·13 + m.
__device__ __forceinline__ int window_flux(const int* bidx, int nb, const Geom& g, int kk, int t) {
    const int comp = kk >= nb, k = comp ? kk - nb : kk, l = t / 13, m = t - 13 * l;
    const int I = bidx[k] + l - 6, J = bidx[nb + k] + m - 6;
    return comp ? g.nu + (I - 1) + (J - 1) * g.nx : (I - 1) + (J - 1) * (g.nx + 1);
}

// The four fluxes of rot! at Γ point (i0, j0): qx[i0+2, j0+1], qx[i0+2, j0+2],
// qy[i0+2, j0+2], qy[i0+1, j0+2] (1-based).
__device__ __forceinline__ void rot_fluxes(const Geom& g, int i0, int j0, int (&f)[4]) {
    f[0] = i0 + 1 + j0 * (g.nx + 1);
    f[1] = f[0] + g.nx + 1;
    f[2] = g.nu + i0 + 1 + (j0 + 1) * g.nx;
    f[3] = f[2] - 1;
}

__global__ void count_kernel(const int* __restrict__ bidx, int nb, Geom g, int* cnt) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < 2 * nb * 169) atomicAdd(cnt + window_flux(bidx, nb, g, e / 169, e % 169), 1);
}

// What item i adds to the scan: a touched flux point one row (high word) and its
// contributors (low word); a Γ point of the source one.
template <bool SRC>
__device__ __forceinline__ unsigned long long scan_item(const int* __restrict__ cnt, const Geom& g, long long i) {
    if (SRC) {
        if (i >= (long long)g.n1 * g.n2) return 0;
        int f[4];
        rot_fluxes(g, (int)(i % g.n1), (int)(i / g.n1), f);
        return (cnt[f[0]] | cnt[f[1]] | cnt[f[2]] | cnt[f[3]]) != 0;
    }
    if (i >= g.nq) return 0;
    const int c = cnt[i];
    return c ? (1ull << 32) + c : 0;
}

// Exclusive sum of v over the block's threads; total to every thread.
__device__ __forceinline__ unsigned long long block_scan(unsigned long long v, unsigned long long& total) {
    __shared__ unsigned long long part[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    unsigned long long s = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long u = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += u;
    }
    if (lane == 31) part[warp] = s;
    __syncthreads();
    unsigned long long before = 0;
    total = 0;
    for (int w = 0; w < nw; ++w) {
        if (w == warp) before = total;
        total += part[w];
    }
    __syncthreads();
    return before + s - v;
}

template <bool SRC>
__global__ void __launch_bounds__(kScanThreads) sums_kernel(const int* __restrict__ cnt, Geom g,
                                                            unsigned long long* sums) {
    unsigned long long v = 0, total;
    const long long i0 = (long long)blockIdx.x * kScanBlock;
#pragma unroll
    for (int r = 0; r < kScanItems; ++r) v += scan_item<SRC>(cnt, g, i0 + r * kScanThreads + threadIdx.x);
    block_scan(v, total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// Exclusive sums of n block sums in place, the total to *total (block 0: the
// fluxes', block 1: the Γ points').
__global__ void __launch_bounds__(1024) offsets_kernel(unsigned long long* fsums, int nf, unsigned long long* ssums,
                                                       int ns, unsigned long long* totals) {
    unsigned long long* s = blockIdx.x ? ssums : fsums;
    const int n = blockIdx.x ? ns : nf;
    unsigned long long carry = 0;
    for (int i0 = 0; i0 < n; i0 += 1024) {
        const int i = i0 + threadIdx.x;
        unsigned long long total;
        const unsigned long long v = i < n ? s[i] : 0, before = block_scan(v, total);
        if (i < n) s[i] = carry + before;
        carry += total;
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

// Each item's place: a flux point's row, its flux and the start of its list
// (row[f] = −1 where untouched), or a Γ point and the rows of its four fluxes.
template <bool SRC>
__global__ void __launch_bounds__(kScanThreads) places_kernel(const int* __restrict__ cnt, Geom g,
                                                              const unsigned long long* __restrict__ sums, int* row,
                                                              CouplingLists c) {
    unsigned long long carry = sums[blockIdx.x];
    const long long i0 = (long long)blockIdx.x * kScanBlock;
    for (int r = 0; r < kScanItems; ++r) {
        const long long i = i0 + r * kScanThreads + threadIdx.x;
        unsigned long long total;
        const unsigned long long v = scan_item<SRC>(cnt, g, i), at = carry + block_scan(v, total);
        carry += total;
        if (SRC) {
            if (!v) continue;
            const int x = (int)(i % g.n1), y = (int)(i / g.n1), p = (int)at;
            int f[4];
            rot_fluxes(g, x, y, f);
            c.src_pts[p] = y * g.P + x;
#pragma unroll
            for (int k = 0; k < 4; ++k) c.src_rows[4 * p + k] = row[f[k]];
        } else if (i < g.nq) {
            const int p = (int)(at >> 32);
            row[i] = v ? p : -1;
            if (!v) continue;
            c.et_flux[p] = (int)i;
            c.et_ptr[p] = (int)at;
            if (p == c.n_rows - 1) c.et_ptr[c.n_rows] = (int)at + (int)v;
        }
    }
}

__global__ void scatter_kernel(const int* __restrict__ bidx, int nb, Geom g, const int* __restrict__ row, int* cnt,
                               CouplingLists c, int* tmp) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= 2 * nb * 169) return;
    const int f = window_flux(bidx, nb, g, e / 169, e % 169);
    tmp[c.et_ptr[row[f]] + atomicSub(cnt + f, 1) - 1] = e / 169;
}

__global__ void rank_kernel(const int* __restrict__ bidx, int nb, Geom g, const int* __restrict__ row,
                            const int* __restrict__ tmp, CouplingLists c) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= 2 * nb * 169) return;
    const int kk = e / 169, r = row[window_flux(bidx, nb, g, kk, e % 169)];
    const int s = c.et_ptr[r], n = c.et_ptr[r + 1] - s;
    int at = s;
#pragma unroll 8
    for (int j = 0; j < n; ++j) at += tmp[s + j] < kk;
    c.et_k[at] = kk;
    c.et_w[at] = e;          // w[kk][l][m]
}

int scan_blocks(long long n) { return (int)((n + kScanBlock - 1) / kScanBlock); }

}  // namespace

// cnt [nq], row [nq], tmp [contributors], then the block sums and the two totals
struct CouplingScratch {
    int *cnt, *row, *tmp;
    unsigned long long *fsums, *ssums, *totals;
    int nfb, nsb;
};

static CouplingScratch scratch_of(const Geom& g, int nb, void* p) {
    CouplingScratch s;
    s.nfb = scan_blocks(g.nq);
    s.nsb = scan_blocks((long long)g.n1 * g.n2);
    s.totals = (unsigned long long*)p;
    s.fsums = s.totals + 2;
    s.ssums = s.fsums + s.nfb;
    s.cnt = (int*)(s.ssums + s.nsb);
    s.row = s.cnt + g.nq;
    s.tmp = s.row + g.nq;
    return s;
}

size_t coupling_scratch_bytes(const Geom& g, int nb) {
    return sizeof(unsigned long long) * (2 + scan_blocks(g.nq) + scan_blocks((long long)g.n1 * g.n2)) +
           sizeof(int) * (2 * (size_t)g.nq + (size_t)nb * 338);
}

cudaError_t launch_coupling_count(const Geom& g, const int* bidx, int nb, void* scratch, cudaStream_t st) {
    const CouplingScratch s = scratch_of(g, nb, scratch);
    cudaError_t e = cudaMemsetAsync(s.cnt, 0, sizeof(int) * (size_t)g.nq, st);
    if (e != cudaSuccess) return e;
    count_kernel<<<(nb * 338 + 255) / 256, 256, 0, st>>>(bidx, nb, g, s.cnt);
    sums_kernel<false><<<s.nfb, kScanThreads, 0, st>>>(s.cnt, g, s.fsums);
    sums_kernel<true><<<s.nsb, kScanThreads, 0, st>>>(s.cnt, g, s.ssums);
    offsets_kernel<<<2, 1024, 0, st>>>(s.fsums, s.nfb, s.ssums, s.nsb, s.totals);
    return cudaGetLastError();
}

cudaError_t launch_coupling_lists(const Geom& g, const int* bidx, int nb, void* scratch, const CouplingLists& c,
                                  cudaStream_t st) {
    const CouplingScratch s = scratch_of(g, nb, scratch);
    const int blocks = (nb * 338 + 255) / 256;
    places_kernel<false><<<s.nfb, kScanThreads, 0, st>>>(s.cnt, g, s.fsums, s.row, c);
    places_kernel<true><<<s.nsb, kScanThreads, 0, st>>>(s.cnt, g, s.ssums, s.row, c);
    scatter_kernel<<<blocks, 256, 0, st>>>(bidx, nb, g, s.row, s.cnt, c, s.tmp);
    rank_kernel<<<blocks, 256, 0, st>>>(bidx, nb, g, s.row, s.tmp, c);
    return cudaGetLastError();
}

}  // namespace ibpm
