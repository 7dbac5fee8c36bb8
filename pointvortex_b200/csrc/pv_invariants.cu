// pv_invariants.cu — invariants of the vortex system on the GPU.
//
// Replaces computeMoments / computeInvariants and the three Hamiltonians of the reference
// (src/compute.cpp:11-27, 134-163, 174-202, 262-285), which the reference evaluates serially on
// the host even with its CUDA backend (src/backend_cuda.cu:245-247).
//
//   * moments: one pass over the vortices, per-thread Neumaier-compensated sums;
//   * Hamiltonian: upper-triangular 128 x 128 tiles of the pair matrix (block b is tile (I, J >= I)
//     with b = J (J + 1) / 2 + I), per-thread compensated sums, per-block (hi, lo) partials. Bound
//     by the FP64 pipe: the pair's energy and its logarithm;
//   * a single-block pass adds the block partials in fixed order, so the result is deterministic
//     and independent of scheduling.
#include "pv_internal.h"
#include "pv_log.cuh"

namespace pvb {

namespace {
constexpr int kHT = 128;                // Hamiltonian tile edge (threads per block)
constexpr int kMomentBlocks = 256;
// Small populations: four (two) blocks share a tile's sources up to 16 (32) tiles an edge, where a
// thread's 128 pairs one after another are the kernel's time (N = 256 to 2048: 16.6 us, with 32 pairs a
// thread 7.5; whole calls, box, plane and disk: N = 1024 61, 56 and 58 us, so 45, 44 and 45; N = 3000 69,
// 57 and 63, so 69, 53 and 57). Returned as a shift.
unsigned tile_split(size_t nt) { return nt <= 16 ? 2 : (nt <= 32 ? 1 : 0); }

// Neumaier's improvement of Kahan summation: s + c carries the sum with the rounding error of
// every addition accumulated in c.
struct CSum {
    double s = 0.0, c = 0.0;
    __device__ __forceinline__ void add(double x) {
        const double t = s + x;
        // the larger first; equal exponents may go either way, so that the high words decide
        const bool first = (__double2hiint(s) & 0x7fffffff) >= (__double2hiint(x) & 0x7fffffff);
        c += ((first ? s : x) - t) + (first ? x : s);
        s = t;
    }
    __device__ __forceinline__ double value() const { return s + c; }
};

__constant__ double c_sech[65];   // 1/cosh(2 pi m), m = 0..64
__constant__ double c_tanh2[65];  // tanh(2 pi m)^2

__device__ __forceinline__ double block_sum_fixed(double v, double *sh) {
    // fixed-order tree: warp shuffles then one warp over the warp sums
    for (int off = 16; off > 0; off >>= 1)
        v += __shfl_down_sync(0xffffffffu, v, off);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0)
        sh[warp] = v;
    __syncthreads();
    double r = 0.0;
    if (warp == 0) {
        r = lane < static_cast<int>(blockDim.x >> 5) ? sh[lane] : 0.0;
        for (int off = 16; off > 0; off >>= 1)
            r += __shfl_down_sync(0xffffffffu, r, off);
    }
    __syncthreads();
    return r;
}

// scratch layout: [0, 4*kMomentBlocks) moment partials (4 per block),
//                 [4*kMomentBlocks, ...) Hamiltonian partials (2 per tile: hi, lo)
__global__ void __launch_bounds__(256)
    moments_kernel(const double *x, const double *y, const double *g, size_t n, double *part,
                   int *status) {
    __shared__ double sh[32];
    CSum c, ix, iy, l;
    bool bad = false;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const double gi = g[i], xi = x[i], yi = y[i];
        if (!isfinite(gi) || !isfinite(xi) || !isfinite(yi))
            bad = true;
        c.add(gi);
        ix.add(gi * xi);
        iy.add(gi * yi);
        l.add(gi * fma(xi, xi, yi * yi));
    }
    if (bad)
        set_status(status, ST_NONFINITE_POSITION);
    const double m0 = block_sum_fixed(c.value(), sh);
    const double m1 = block_sum_fixed(ix.value(), sh);
    const double m2 = block_sum_fixed(iy.value(), sh);
    const double m3 = block_sum_fixed(l.value(), sh);
    if (threadIdx.x == 0) {
        part[4 * blockIdx.x + 0] = m0;
        part[4 * blockIdx.x + 1] = m1;
        part[4 * blockIdx.x + 2] = m2;
        part[4 * blockIdx.x + 3] = m3;
    }
}

// Pair energies (the sum that the reference multiplies by -1/(4 pi)):
//   infinite: G_i G_j log(r^2 + eps^2)
//   periodic: G_i G_j [ -x^2/(2 pi) + log D_0 + log prod_{m=1..M} D_m D_-m / cosh^2(2 pi m) ]
//             with D_m D_-m / cosh^2 a = (cosh x^ sech a - cos y^)^2 + tanh^2 a sin^2 y^, which is
//             the reference's sum over m of log(den_m) - logCosh(2 pi m) (src/compute.cpp:186-196)
//   disk:     G_i G_j log(|z_i - z_j|^2 R^2 / ((R^2 - z_i.z_j)^2 + (z_i x z_j)^2))
// plus, for the disk, the self terms -G_i^2 log((R^2 - r_i^2)/R) (entered with the sign that makes
// the final -sum/(4 pi) equal the reference).
//
// ZETA: the box from six images up by box_energy (pv_geometry.cuh).
//
// A pair's energy is the logarithm of an argument, plus `rest` for the box. Each thread sums its pairs
// with log_normal (pv_log.cuh), without a branch, and notes whether an argument was not a positive normal
// number (coincident, overflowed, beyond the reach of the reduction); then it sums them again with
// energy(), which handles and reports all that. stateInvariants at N = 65 536 with the library's
// logarithm and division, which branch, and so: box 13.0 and 8.6 ms, plane 8.0 and 4.5, disk 10.3 and
// 6.2; the pairs' FP64 instructions (box 50, plane 22, disk 33) alone take 5.8, 2.5 and 3.8 ms. Errors
// against 80-bit sums, rms over 150 populations of 250, in units of the terms' 2-norm: plane 1.9e-16
// both, disk 2.0e-16 both, box 6.4e-15 with the image product and 2.7e-15.
// EXACT: the disk's quotient by division; else by a reciprocal and one residual, without a branch, which
// is as good wherever the result and its operands are normal numbers, and 0, infinite or NaN elsewhere.
template <int GEO, bool ZETA, bool EXACT>
__device__ __forceinline__ double argument(const GeometryConsts &gc, double xi, double yi, double xj,
                                           double yj, bool near, double &rest) {
    rest = 0.0;
    const double dx = xi - xj, dy = yi - yj;
    if (GEO == GEO_INFINITE)
        return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), gc.eps2);
    if (ZETA)
        return near ? box_energy(gc, ZetaPair::reduce_near(gc, dx, gc.lx),
                                 ZetaPair::reduce_near(gc, dy, gc.ly), rest)
                    : box_energy(gc, ZetaPair::reduce(gc, dx, gc.lx, gc.inv_lx),
                                 ZetaPair::reduce(gc, dy, gc.ly, gc.inv_ly), rest);
    const double num = (dx * dx + dy * dy) * gc.radius2;
    const double dot = xi * xj + yi * yj;
    const double cross = yi * xj - xi * yj;
    const double den = (gc.radius2 - dot) * (gc.radius2 - dot) + cross * cross;
    if (EXACT)
        return num / den;
    const double inv = rcp_refined(den);
    const double q = num * inv;
    return fma(fma(-q, den, num), inv, q);
}

template <int GEO, bool ZETA>
__device__ __forceinline__ double energy(const GeometryConsts &gc, double xi, double yi, double xj,
                                      double yj, int *status) {
    if (GEO != GEO_PERIODIC) {
        double rest;
        const double a = argument<GEO, ZETA, true>(gc, xi, yi, xj, yj, false, rest);
        // the disk's argument is 0 as well where its numerator only vanishes against the denominator
        if (GEO == GEO_INFINITE ? a == 0.0
                                : ((xi - xj) * (xi - xj) + (yi - yj) * (yi - yj)) * gc.radius2 == 0.0)
            set_status(status, ST_COINCIDENT);
        return log(a);
    }
    if (ZETA) {
        double rest;
        const double x = ZetaPair::reduce_any(gc, xi - xj, gc.lx, gc.inv_lx);
        const double y = ZetaPair::reduce_any(gc, yi - yj, gc.ly, gc.inv_ly);
        const double a = box_energy(gc, x, y, rest);
        if (fma(x, x, y * y) == 0.0)
            set_status(status, ST_COINCIDENT);
        return rest + log(a);
    }
    const double xh = gc.wave * exact_remainder(xi - xj, gc.lx, gc.inv_lx, gc.half_lx);
    const double yh = gc.wave * exact_remainder(yi - yj, gc.ly, gc.inv_ly, gc.half_ly);
    double shx, chx, snx, csx, shy, chy, sny, csy;
    sinh_cosh_sin_cos(0.5 * xh, shx, chx, snx, csx);
    sinh_cosh_sin_cos(0.5 * yh, shy, chy, sny, csy);
    const double d0 = 2.0 * fma(shx, shx, sny * sny);
    if (d0 == 0.0)
        set_status(status, ST_COINCIDENT);
    const double cosh_x = fma(2.0 * shx, shx, 1.0);
    const double cos_y = fma(-2.0 * sny, sny, 1.0);
    const double sin_y = 2.0 * sny * csy;
    const double s2 = sin_y * sin_y;
    double prod = 1.0;
    for (int m = 1; m <= gc.image_layers; ++m) {
        const double q = fma(cosh_x, c_sech[m], -cos_y);
        prod *= fma(q, q, c_tanh2[m] * s2);
    }
    return -xh * xh / (2.0 * kPi) + log(d0) + log(prod);
}

// The pairs of vortex i with [jstart, jcount) of the tile; false where an argument was irregular.
template <int GEO, bool ZETA, bool NEAR>
__device__ __forceinline__ bool regular_pairs(const GeometryConsts &gc, double xi, double yi,
                                              const double *sx, const double *sy, const double *sg,
                                              const LogPoint *table, int jstart, int jcount,
                                              CSum &acc) {
    bool regular = true;
#pragma unroll 4
    for (int jj = jstart; jj < jcount; ++jj) {
        double rest;
        const double a = argument<GEO, ZETA, false>(gc, xi, yi, sx[jj], sy[jj], NEAR, rest);
        regular = regular && log_is_normal(a);
        const double l = log_normal(a, table);
        acc.add(sg[jj] * (ZETA ? rest + l : l));
    }
    return regular;
}

template <int GEO, bool ZETA = false>
__global__ void __launch_bounds__(kHT)
    hamiltonian_kernel(const double *x, const double *y, const double *g, size_t n,
                       GeometryConsts gc, unsigned split, double *part, int *status) {
    pdl_enter();
    const unsigned tile_index = blockIdx.x >> split, share = blockIdx.x & ((1u << split) - 1);
    unsigned J = static_cast<unsigned>((sqrt(8.0 * tile_index + 1.0) - 1.0) * 0.5);
    while (static_cast<unsigned long long>(J + 1) * (J + 2) / 2 <= tile_index)
        ++J;
    while (static_cast<unsigned long long>(J) * (J + 1) / 2 > tile_index)
        --J;
    const unsigned I = tile_index - J * (J + 1) / 2;
    constexpr bool kRegular = GEO != GEO_PERIODIC || ZETA;  // the form has a loop without branches
    __shared__ double sx[kHT], sy[kHT], sg[kHT];
    __shared__ double sh[32];
    __shared__ LogPoint table[kRegular ? kLogPoints : 1];
    if (kRegular)
        for (int k = threadIdx.x; k < kLogPoints; k += kHT)
            table[k] = kLogTable[k];
    CSum acc;          // the pairs' energies times the other vortex's circulation
    double gi = 0.0;
    const size_t i = static_cast<size_t>(I) * kHT + threadIdx.x;
    const size_t j0 = static_cast<size_t>(J) * kHT;
    const size_t jl = j0 + threadIdx.x;
    sx[threadIdx.x] = jl < n ? x[jl] : 0.0;
    sy[threadIdx.x] = jl < n ? y[jl] : 0.0;
    sg[threadIdx.x] = jl < n ? g[jl] : 0.0;
    const double xi = i < n ? x[i] : 0.0, yi = i < n ? y[i] : 0.0;
    bool near = true;
    if (ZETA)
        near = __syncthreads_and(ZetaPair::inside(gc, xi, yi) &&
                                 ZetaPair::inside(gc, sx[threadIdx.x], sy[threadIdx.x]));
    else
        __syncthreads();
    if (i < n) {
        gi = g[i];
        const int sources = kHT >> split, first = static_cast<int>(share) * sources;
        const int jcount = static_cast<int>(min(static_cast<size_t>(first + sources), n - j0));
        const int jstart = max(first, (I == J) ? static_cast<int>(threadIdx.x) + 1 : 0);
        bool done = false;
        if (kRegular)
            done = near ? regular_pairs<GEO, ZETA, true>(gc, xi, yi, sx, sy, sg, table, jstart, jcount,
                                                         acc)
                        : regular_pairs<GEO, ZETA, false>(gc, xi, yi, sx, sy, sg, table, jstart,
                                                          jcount, acc);
        if (!done) {
            acc = CSum();
            for (int jj = jstart; jj < jcount; ++jj)
                acc.add(sg[jj] * energy<GEO, ZETA>(gc, xi, yi, sx[jj], sy[jj], status));
        }
        if (GEO == GEO_DISK && I == J && share == 0) {
            const double ri2 = __dadd_rn(__dmul_rn(xi, xi), __dmul_rn(yi, yi));
            if (ri2 >= gc.radius2)
                set_status(status, ST_OUTSIDE_DISK_H);
            acc.add(-gi * log(__ddiv_rn(gc.radius2 - ri2, gc.radius)));
        }
    }
    const double hi = block_sum_fixed(gi * acc.s, sh);
    const double lo = block_sum_fixed(gi * acc.c, sh);
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = hi;
        part[2 * blockIdx.x + 1] = lo;
    }
}

// One block: fixed-order compensated sums of the moment partials (a warp each) and of the Hamiltonian
// partials.
__global__ void __launch_bounds__(1024)
    finalize_kernel(const double *part, int moment_blocks, size_t tiles, double *out, int *status,
                    int *status_h) {
    pdl_enter();
    __shared__ double sh[32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp < 4) {
        CSum c;
#pragma unroll 8
        for (int b = lane; b < moment_blocks; b += 32)
            c.add(part[4 * b + warp]);
        double hi = c.s, lo = c.c;
        for (int off = 16; off > 0; off >>= 1) {
            hi += __shfl_down_sync(0xffffffffu, hi, off);
            lo += __shfl_down_sync(0xffffffffu, lo, off);
        }
        if (lane == 0) {
            out[warp] = hi + lo;
            if (!isfinite(hi + lo))
                set_status_if_clean(status, ST_NONFINITE_MOMENT);
        }
    }
    const double *hp = part + 4 * moment_blocks;
    CSum h;
    for (size_t t = threadIdx.x; t < tiles; t += blockDim.x) {
        h.add(hp[2 * t]);
        h.add(hp[2 * t + 1]);
    }
    const double hi = block_sum_fixed(h.s, sh);
    const double lo = block_sum_fixed(h.c, sh);
    if (threadIdx.x == 0) {
        const double hamiltonian = -(hi + lo) / (4.0 * kPi);
        out[4] = hamiltonian;
        if (!isfinite(hamiltonian))
            set_status_if_clean(status_h, ST_NONFINITE_HAMILTONIAN);
    }
}

bool g_tables_ready[64] = {};
} // namespace

size_t invariants_scratch_doubles(size_t n, int) {
    const size_t nt = (n + kHT - 1) / kHT;
    return 4 * static_cast<size_t>(kMomentBlocks) +
           2 * (nt > 0 ? (nt * (nt + 1) / 2) << tile_split(nt) : 1);
}

cudaError_t launch_invariants(const double *x, const double *y, const double *gamma, size_t n,
                              const GeometryConsts &g, double *scratch, double *out, int *status,
                              int *status_h, cudaStream_t stream) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (g.geometry == GEO_PERIODIC && dev >= 0 && dev < 64 && !g_tables_ready[dev]) {
        double sech[65], tanh2[65];
        for (int m = 0; m <= 64; ++m) {
            const double a = 2.0 * kPi * m;
            sech[m] = 1.0 / cosh(a);
            const double t = tanh(a);
            tanh2[m] = t * t;
        }
        cudaError_t e = cudaMemcpyToSymbol(c_sech, sech, sizeof(sech));
        if (e == cudaSuccess)
            e = cudaMemcpyToSymbol(c_tanh2, tanh2, sizeof(tanh2));
        if (e != cudaSuccess)
            return e;
        g_tables_ready[dev] = true;
    }
    moments_kernel<<<kMomentBlocks, 256, 0, stream>>>(x, y, gamma, n, scratch, status);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return e;
    const size_t nt = (n + kHT - 1) / kHT;
    size_t tiles = 0;
    if (nt > 0) {
        const unsigned split = tile_split(nt);
        tiles = (nt * (nt + 1) / 2) << split;
        if (tiles > 0x7fffffffu)
            return cudaErrorInvalidValue;
        const dim3 grid(static_cast<unsigned>(tiles));
        double *hp = scratch + 4 * kMomentBlocks;
        switch (g.geometry) {
        case GEO_INFINITE:
            e = launch_pdl(hamiltonian_kernel<GEO_INFINITE>, grid, dim3(kHT), 0, stream, x, y, gamma,
                           n, g, split, hp, status_h);
            break;
        case GEO_PERIODIC:
            e = g.zeta ? launch_pdl(hamiltonian_kernel<GEO_PERIODIC, true>, grid, dim3(kHT), 0,
                                    stream, x, y, gamma, n, g, split, hp, status_h)
                       : launch_pdl(hamiltonian_kernel<GEO_PERIODIC>, grid, dim3(kHT), 0, stream, x,
                                    y, gamma, n, g, split, hp, status_h);
            break;
        default:
            e = launch_pdl(hamiltonian_kernel<GEO_DISK>, grid, dim3(kHT), 0, stream, x, y, gamma, n,
                           g, split, hp, status_h);
            break;
        }
        if (e != cudaSuccess)
            return e;
    }
    return launch_pdl(finalize_kernel, dim3(1), dim3(1024), 0, stream, scratch, kMomentBlocks, tiles,
                      out, status, status_h);
}

} // namespace pvb
