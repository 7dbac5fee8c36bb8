// pv_stepping.cu — the Runge–Kutta stage work between two velocity evaluations, on the GPU.
//
// Replaces RungeKuttaIntegrator::makeStage / rk4Step / dopri5Step (src/timestep.cpp:19-120)
// and the reference CUDA backend's stage, combine, validation and error kernels with their
// host round trips (src/backend_cuda.cu:115-200, 299-357, 387-450). One kernel per stage:
//
//   1. reduce the evaluation's chunk partials into k_s in fixed chunk order; a target whose sum is
//      non-finite is recomputed in the reference form (IEEE divisions, the reference's singular
//      test), which either yields the reference's finite value or its error;
//   2. per mode: the next stage position y0 + dt * sum_j a_j k_j, or the RK4 combination, or the
//      DOPRI5 scaled error (max-reduced with one atomicMax per block), each validated like the
//      reference (finite positions; in a disk, inside the wall);
//   3. DOPRI5: the last block to finish runs the step-size control of src/timestep.cpp:97-118 on
//      the device (accept/reject, suggested step, rejection cap), so the state never leaves the GPU
//      between attempts.
//
// All combination arithmetic uses explicitly rounded operations (__dmul_rn/__dadd_rn/__ddiv_rn)
// in the reference's order, so that given the same stage velocities the new state is bit-identical
// to the reference's (which x86-64 g++ computes without FMA contraction).
#include "pv_barrier.cuh"
#include "pv_internal.h"

#include <algorithm>
#include <type_traits>

namespace pvb {

namespace {
__device__ __forceinline__ double max_ref(double a, double b) { return (a < b) ? b : a; }
__device__ __forceinline__ double min_ref(double a, double b) { return (b < a) ? b : a; }
__device__ __forceinline__ double clamp_ref(double v, double lo, double hi) {
    return v < lo ? lo : (hi < v ? hi : v);
}

// Verdict on a new position (0: valid), src/vortex.h:7-14 and src/compute.cpp:41-48.
__device__ __forceinline__ int position_error(const GeometryConsts &g, double x, double y) {
    if (!isfinite(x) || !isfinite(y))
        return ST_NONFINITE_POSITION;
    if (g.geometry == GEO_DISK && __dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)) >= g.radius2)
        return ST_OUTSIDE_DISK;
    return 0;
}

__device__ __forceinline__ void validate_position(const StageArgs &a, double x, double y) {
    const int e = position_error(a.g, x, y);
    if (e)
        set_status(&a.ctl->status, e);
}

// src/timestep.cpp:52-57: x0 + dt * (k1 + 2 k2 + 2 k3 + k4) / 6
__device__ __forceinline__ double rk4_point(double x0, double dt, double k1, double k2, double k3,
                                            double k4) {
    const double s = __dadd_rn(
        __dadd_rn(__dadd_rn(k1, __dmul_rn(2.0, k2)), __dmul_rn(2.0, k3)), k4);
    return __dadd_rn(x0, __ddiv_rn(__dmul_rn(dt, s), 6.0));
}

// The scale of an error component, src/timestep.cpp:84-87.
__device__ __forceinline__ double error_scale(const DeviceControl *ctl, double x0, double x5) {
    return __dadd_rn(ctl->absolute_tolerance,
                     __dmul_rn(ctl->relative_tolerance, max_ref(fabs(x0), fabs(x5))));
}

// DOPRI5 step-size control, src/timestep.cpp:95-118. Returns ST_DOPRI_FAILED, or 0.
__device__ __forceinline__ int dopri_decide(double error, double dt, double minimum,
                                            double maximum, unsigned &rejected, int &accepted,
                                            double &suggested, double &next_dt) {
    const double factor = error == 0.0 ? 5.0 : clamp_ref(0.9 * pow(error, -0.2), 0.2, 5.0);
    suggested = clamp_ref(__dmul_rn(dt, factor), minimum, maximum);
    next_dt = dt;
    accepted = error <= 1.0 ? 1 : 0;
    if (accepted)
        return 0;
    if (dt <= minimum || ++rejected > 32u)
        return ST_DOPRI_FAILED;
    next_dt = max_ref(minimum, min_ref(suggested, __dmul_rn(dt, 0.9)));
    return 0;
}

__device__ __forceinline__ void store_accepted(DeviceControl *ctl, double dt, double suggested,
                                               double error, unsigned rejected) {
    ctl->result[0] = dt;
    ctl->result[1] = suggested;
    ctl->result[2] = error;
    ctl->result[3] = static_cast<double>(rejected);
}

// The control of an attempt made by launches, run by one thread.
__device__ void dopri_control(DeviceControl *ctl) {
    const double error = __longlong_as_double(static_cast<long long>(ctl->err_bits));
    const double dt = ctl->dt;
    if (ctl->status == 0) {
        double suggested, next_dt;
        unsigned rejected = ctl->rejected;
        int accepted;
        const int failed = dopri_decide(error, dt, ctl->minimum_time_step, ctl->maximum_time_step,
                                        rejected, accepted, suggested, next_dt);
        ctl->accepted = accepted;
        ctl->rejected = rejected;
        ctl->dt = next_dt;
        if (accepted)
            store_accepted(ctl, dt, suggested, error, rejected);
        if (failed)
            set_status(&ctl->status, failed);
    }
    ctl->err_bits = 0ull;
    ctl->blocks_done = 0u;
    ctl->dipole_count = 0ull;  // the attempt's gated dipole scan counts from here
}
} // namespace

// What a target's finish reads besides its own velocity: the step-start position, the earlier
// stage velocities k_j (j != s) that its combination uses, and for the DOPRI5 error the
// fifth-order point. All of them were written by kernels that completed before this stage kernel
// was launched (the earlier stage kernels; the velocity launch it waits for writes only partial
// rows), so the stage kernel may load them before its wait on the velocity launch.
struct FinishInputs {
    double x0, y0, xt, yt;
    double kx[7], ky[7];
};

template <int MODE>
__device__ __forceinline__ void load_finish_inputs(const StageArgs &a, size_t i, FinishInputs &p) {
    p.x0 = a.x0[i];
    p.y0 = a.y0[i];
    if (MODE == STAGE_DOPRI_ERROR) {
        p.xt = a.xt[i];
        p.yt = a.yt[i];
    }
#pragma unroll
    for (int j = 0; j < 7; ++j) {
        bool used = false;
        if (MODE == STAGE_POSITION)
            used = j < a.ncoef && a.coef[j] != 0.0;
        else if (MODE == STAGE_DOPRI_ERROR)
            used = a.w[j] != 0.0;
        else if (MODE == STAGE_RK4_COMBINE)
            used = j < 3;
        if (used && j != a.s) {
            p.kx[j] = a.kx[j][i];
            p.ky[j] = a.ky[j][i];
        }
    }
}

// Everything a stage does for one target once its velocity (ku, kv) is summed: the slow path of
// a non-finite sum, the stage velocity, and the stage position / RK4 combination / DOPRI5 error.
// ex, ey: the positions the slow path recomputes from (a.ex, a.ey, or a copy of them). p: the
// target's FinishInputs.
template <int MODE>
__device__ __forceinline__ void finish_target(const StageArgs &a, size_t i, double ku, double kv,
                                              double dt, double &local_max, const double *ex,
                                              const double *ey, const FinishInputs &p) {
    if (a.reduce) {
        if (!isfinite(ku) || !isfinite(kv)) {
            const int verdict =
                slow_target(a.g, ex, ey, a.gamma, a.n_src, a.t_offset + i, ku, kv);
            if (verdict == ST_COINCIDENT || (verdict && !a.nonfinite_ok))
                set_status(&a.ctl->status, verdict);
        }
        a.kx[a.s][i] = ku;
        a.ky[a.s][i] = kv;
    }
    if (MODE == STAGE_POSITION) {
        // makeStage, src/timestep.cpp:19-30 (zero coefficients add an exact zero: skipped)
        double dx = 0.0, dy = 0.0;
#pragma unroll
        for (int j = 0; j < 7; ++j) {  // unrolled: p's fields stay in registers
            const double c = a.coef[j];
            if (j >= a.ncoef || c == 0.0)
                continue;
            const double kxj = j == a.s ? ku : p.kx[j];
            const double kyj = j == a.s ? kv : p.ky[j];
            dx = __dadd_rn(dx, __dmul_rn(c, kxj));
            dy = __dadd_rn(dy, __dmul_rn(c, kyj));
        }
        const double nx = __dadd_rn(p.x0, __dmul_rn(dt, dx));
        const double ny = __dadd_rn(p.y0, __dmul_rn(dt, dy));
        a.xt[i] = nx;
        a.yt[i] = ny;
        validate_position(a, nx, ny);
    } else if (MODE == STAGE_RK4_COMBINE) {
        const double nx = rk4_point(p.x0, dt, p.kx[0], p.kx[1], p.kx[2], ku);
        const double ny = rk4_point(p.y0, dt, p.ky[0], p.ky[1], p.ky[2], kv);
        a.xt[i] = nx;
        a.yt[i] = ny;
        if (!isfinite(nx) || !isfinite(ny))
            set_status(&a.ctl->status, ST_NONFINITE_POSITION);
    } else if (MODE == STAGE_DOPRI_ERROR) {
        // src/timestep.cpp:78-95: xt holds the fifth-order point y5 (stage 7's position).
        double xe = 0.0, ye = 0.0;
#pragma unroll
        for (int j = 0; j < 7; ++j) {
            const double w = a.w[j];
            if (w == 0.0)
                continue;
            const double h = __dmul_rn(dt, w);
            const double kxj = j == a.s ? ku : p.kx[j];
            const double kyj = j == a.s ? kv : p.ky[j];
            xe = __dadd_rn(xe, __dmul_rn(h, kxj));
            ye = __dadd_rn(ye, __dmul_rn(h, kyj));
        }
        const double x5 = p.xt, y5 = p.yt;
        const double xs = error_scale(a.ctl, p.x0, x5), ys = error_scale(a.ctl, p.y0, y5);
        if (!isfinite(xe) || !isfinite(ye) || !isfinite(xs) || !isfinite(ys) || !(xs > 0.0) ||
            !(ys > 0.0)) {
            set_status(&a.ctl->status, ST_DOPRI_NONFINITE);
        } else {
            local_max = max_ref(local_max, __ddiv_rn(fabs(xe), xs));
            local_max = max_ref(local_max, __ddiv_rn(fabs(ye), ys));
        }
    }
}

// The near-field terms of the block's kWideTargets targets, fused into the wide stage (the work of
// pv_near.cu's near_field_kernel): the kWideGroups threads of a target share its listed entries
// (at most f32::kNearSlots), each computes its entries' FP64 terms (the plain kernels' pair
// functions) and their rank in (source, image) order, and the target's first thread adds them in
// that order, so the sum does not depend on the order of the listing. A target with more
// entries than slots is evaluated whole in FP64 instead (every thread of the block striding over the
// sources, their sums added in a fixed tree), replacing its partial rows. One such target among
// N = 12 000 makes the stage 469 us when only its own 16 threads share it, 41 us so. Every
// count is reset.
// Returns, for the calling first thread (group 0) of target `lane`, the near sum (nu, nv) and
// whether it replaces the rows.
struct NearScratch {
    unsigned key[16][f32::kNearSlots];
    double tu[16][f32::kNearSlots], tv[16][f32::kNearSlots];
    int over[16];             // targets evaluated whole
    double warp_u[8], warp_v[8];
};

__device__ __forceinline__ bool fused_near(const NearPass &np, size_t i, bool valid, int lane,
                                           int group, int groups, NearScratch &sc, double &nu,
                                           double &nv) {
    const size_t gi = np.t_begin + i;
    // every thread of the target reads its count (the first one resets it after the barrier
    // below, once all have read it)
    const unsigned count = valid ? np.lists.count[gi] : 0u;
    const bool whole = count > static_cast<unsigned>(f32::kNearSlots);
    nu = nv = 0.0;
    const double tx = valid && count ? np.x[gi] : 0.0, ty = valid && count ? np.y[gi] : 0.0;
    if (group == 0)
        sc.over[lane] = whole ? 1 : 0;
    if (!whole && count) {
        for (int e = group; e < static_cast<int>(count); e += groups) {
            const unsigned v = np.lists.slot[gi * f32::kNearSlots + e];
            sc.key[lane][e] = (v & ~f32::kNearImage) * 2u + (v >> 31);
        }
    }
    const int any_over = __syncthreads_or(whole);
    if (group == 0 && count)
        np.lists.count[gi] = 0u;
    if (any_over) {
        const size_t first = gi - static_cast<size_t>(lane);  // the block's first target
        for (int l = 0; l < 16; ++l) {
            if (!sc.over[l])  // the same answer in every thread
                continue;
            const size_t t = first + l;
            const double px = np.x[t], py = np.y[t];
            double su = 0.0, sv = 0.0;
            for (size_t j = threadIdx.x; j < np.n; j += blockDim.x) {
                if (np.g.geometry == GEO_PERIODIC)
                    periodic_pair<true>(np.g, px, py, np.x[j], np.y[j], np.gs[j], j == t, su, sv);
                else
                    DiskPair::pair<true>(np.g, px, py, np.x[j], np.y[j], np.gs[j], j == t, su, sv);
            }
            for (int off = 16; off > 0; off >>= 1) {
                su += __shfl_down_sync(0xffffffffu, su, off);
                sv += __shfl_down_sync(0xffffffffu, sv, off);
            }
            if ((threadIdx.x & 31) == 0) {
                sc.warp_u[threadIdx.x >> 5] = su;
                sc.warp_v[threadIdx.x >> 5] = sv;
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                for (int w = 1; w < 8; ++w) {
                    su += sc.warp_u[w];
                    sv += sc.warp_v[w];
                }
                sc.tu[l][0] = su;
                sc.tv[l][0] = sv;
            }
            __syncthreads();
        }
    }
    if (!whole && count) {
        for (int e = group; e < static_cast<int>(count); e += groups) {
            const unsigned key = sc.key[lane][e];
            int rank = 0;
            for (int k = 0; k < static_cast<int>(count); ++k)
                rank += sc.key[lane][k] < key ? 1 : 0;
            double du = 0.0, dv = 0.0;
            const size_t j = key >> 1;
            if (key & 1u)
                DiskPair::image(np.g, tx, ty, np.x[j], np.y[j], np.gs[j], du, dv);
            else if (np.g.geometry == GEO_PERIODIC)
                periodic_pair<false>(np.g, tx, ty, np.x[j], np.y[j], np.gs[j], false, du, dv);
            else
                DiskPair::direct(tx, ty, np.x[j], np.y[j], np.gs[j], du, dv);
            sc.tu[lane][rank] = du;
            sc.tv[lane][rank] = dv;
        }
    }
    __syncthreads();
    if (group == 0 && count) {
        const int terms = whole ? 1 : static_cast<int>(count);
        for (int r = 0; r < terms; ++r) {
            nu += sc.tu[lane][r];
            nv += sc.tv[lane][r];
        }
    }
    return whole;
}

// Fewer than kWideRows rows: four interleaved sums (rows 0, 4, 8, ...; 1, 5, ...), so that a chain of
// dependent additions is a quarter of the rows long, and four rows are in flight. The cooperative
// steps add their chunks in the same order.
template <class Row>
__device__ __forceinline__ void sum_chunks(int rows, Row &&row, double &ku, double &kv) {
    double u[4] = {0.0, 0.0, 0.0, 0.0}, v[4] = {0.0, 0.0, 0.0, 0.0};
    for (int c = 0; c < rows; c += 4) {
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (c + q < rows) {
                double ru, rv;
                row(c + q, ru, rv);
                u[q] += ru;
                v[q] += rv;
            }
    }
    ku = (u[0] + u[1]) + (u[2] + u[3]);
    kv = (v[0] + v[1]) + (v[2] + v[3]);
}

// WIDE: many partial rows (the symmetric kernel's). A block then covers kWideTargets targets with
// 256 / kWideTargets row groups: thread (group, t) sums rows group, group + groups, ...
// (coalesced over the targets), and the threads of group 0 add the group sums in fixed order.
// Otherwise one thread per target sums its rows in order.
constexpr int kWideTargets = 16;
constexpr int kWideGroups = 256 / kWideTargets;

template <int MODE, bool WIDE, bool NEAR = false>
__global__ void __launch_bounds__(256) stage_kernel(const StageArgs a) {
    __shared__ int s_status;
    __shared__ double s_max[8];
    __shared__ double s_u[WIDE ? kWideGroups : 1][kWideTargets],
        s_v[WIDE ? kWideGroups : 1][kWideTargets];
    __shared__ typename std::conditional<NEAR, NearScratch, char>::type s_near;
    const int tid = threadIdx.x;
    // WIDE: the finishing threads load their first target's FinishInputs before the wait
    FinishInputs early;
    const size_t first = static_cast<size_t>(blockIdx.x) * kWideTargets + tid % kWideTargets;
    if (WIDE && tid < kWideTargets && first < a.n && MODE != STAGE_REDUCE_ONLY)
        load_finish_inputs<MODE>(a, first, early);
    pdl_enter();
    if (tid == 0)
        s_status = *reinterpret_cast<volatile int *>(&a.ctl->status);
    __syncthreads();
    if (s_status != 0) {
        if (NEAR)  // the next evaluation starts from empty lists
            for (size_t i = static_cast<size_t>(blockIdx.x) * kWideTargets + tid; i < a.n;
                 i += static_cast<size_t>(gridDim.x) * kWideTargets)
                if (tid < kWideTargets)
                    a.near.lists.count[a.near.t_begin + i] = 0u;
        return;
    }

    const double dt = a.dt_from_control ? a.ctl->dt : a.dt;
    double local_max = 0.0;
    if (WIDE) {
        const int lane = tid % kWideTargets, group = tid / kWideTargets;
        for (size_t base = static_cast<size_t>(blockIdx.x) * kWideTargets; base < a.n;
             base += static_cast<size_t>(gridDim.x) * kWideTargets) {
            const size_t i = base + lane;
            double su = 0.0, sv = 0.0;
            if (i < a.n && a.pr) {
                // interleaved rows: one 16-byte load per row, eight rows in flight per thread
                // before they are added (in row order, so the sum does not depend on timing)
                const double2 *col = a.pr + i;
                const size_t step = static_cast<size_t>(kWideGroups) * a.stride;
                int c = group;
                for (; c + 7 * kWideGroups < a.num_chunks; c += 8 * kWideGroups) {
                    double2 r[8];
                    const double2 *p = col + static_cast<size_t>(c) * a.stride;
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        r[q] = __ldcg(p + q * step);
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        su += r[q].x;
                        sv += r[q].y;
                    }
                }
                for (; c < a.num_chunks; c += kWideGroups) {
                    const double2 r = __ldcg(col + static_cast<size_t>(c) * a.stride);
                    su += r.x;
                    sv += r.y;
                }
            } else if (i < a.n) {
                for (int c = group; c < a.num_chunks; c += kWideGroups) {
                    su += a.pu[static_cast<size_t>(c) * a.stride + i];
                    sv += a.pv[static_cast<size_t>(c) * a.stride + i];
                }
            }
            s_u[group][lane] = su;
            s_v[group][lane] = sv;
            double nu = 0.0, nv = 0.0;
            bool whole = false;
            if constexpr (NEAR)  // its barriers also order the row sums above
                whole = fused_near(a.near, i, i < a.n, lane, group, kWideGroups, s_near, nu, nv);
            __syncthreads();
            if (group == 0 && i < a.n) {
                double ku = s_u[0][lane], kv = s_v[0][lane];
                for (int g = 1; g < kWideGroups; ++g) {
                    ku += s_u[g][lane];
                    kv += s_v[g][lane];
                }
                if (NEAR) {  // the near terms after the rows, or instead of them
                    ku = whole ? nu : ku + nu;
                    kv = whole ? nv : kv + nv;
                }
                if (i != first && MODE != STAGE_REDUCE_ONLY)
                    load_finish_inputs<MODE>(a, i, early);
                finish_target<MODE>(a, i, ku, kv, dt, local_max, a.ex, a.ey, early);
            }
            __syncthreads();
        }
    } else {
        for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + tid; i < a.n;
             i += static_cast<size_t>(gridDim.x) * blockDim.x) {
            double ku, kv;
            if (a.reduce) {
                const auto row = [&](int c, double &ru, double &rv) {
                    if (a.pr) {
                        const double2 r = a.pr[static_cast<size_t>(c) * a.stride + i];
                        ru = r.x;
                        rv = r.y;
                    } else {
                        ru = a.pu[static_cast<size_t>(c) * a.stride + i];
                        rv = a.pv[static_cast<size_t>(c) * a.stride + i];
                    }
                };
                sum_chunks(a.num_chunks, row, ku, kv);
            } else {
                ku = a.kx[a.s][i];
                kv = a.ky[a.s][i];
            }
            FinishInputs in;
            if (MODE != STAGE_REDUCE_ONLY)
                load_finish_inputs<MODE>(a, i, in);
            finish_target<MODE>(a, i, ku, kv, dt, local_max, a.ex, a.ey, in);
        }
    }

    if (MODE == STAGE_DOPRI_ERROR) {
        // Block max (max is exact, so the order of the reduction cannot change the result).
        for (int off = 16; off > 0; off >>= 1)
            local_max = max_ref(local_max, __shfl_xor_sync(0xffffffffu, local_max, off));
        if ((tid & 31) == 0)
            s_max[tid >> 5] = local_max;
        __syncthreads();
        if (tid == 0) {
            double m = 0.0;
            for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w)
                m = max_ref(m, s_max[w]);
            atomicMax(&a.ctl->err_bits, ordered_bits(m));
            __threadfence();
            const unsigned done = atomicAdd(&a.ctl->blocks_done, 1u);
            if (done == gridDim.x - 1) {
                __threadfence();
                dopri_control(a.ctl);
            }
        }
    }
}

__global__ void __launch_bounds__(256)
    accept_kernel(double *x, double *y, const double *xt, const double *yt, double *k0x,
                  double *k0y, const double *k6x, const double *k6y, size_t n, int dopri,
                  const DeviceControl *ctl) {
    pdl_enter();
    if (ctl->status != 0 || (dopri && !ctl->accepted))
        return;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        x[i] = xt[i];
        y[i] = yt[i];
        if (dopri) { // FSAL: k7 of the accepted step is k1 of the next (src/timestep.cpp:104-108)
            k0x[i] = k6x[i];
            k0y[i] = k6y[i];
        }
    }
}

namespace {
unsigned grid_for(size_t n, int sm_count) {
    const size_t blocks = (n + 255) / 256;
    const size_t cap = static_cast<size_t>(sm_count > 0 ? sm_count : 148) * 8;
    return static_cast<unsigned>(blocks < 1 ? 1 : (blocks < cap ? blocks : cap));
}
} // namespace

// Partial rows from which a block of 32 targets x 8 row groups beats one thread per target.
constexpr int kWideRows = 32;

template <int MODE>
cudaError_t launch_stage_mode(const StageArgs &a, cudaStream_t stream, int sm_count) {
    const bool near = a.near.lists.count != nullptr;
    if (near && !a.reduce)
        return cudaErrorInvalidValue;
    // the near-field terms need the wide layout (a target's threads share its list), whatever
    // the number of rows
    if (a.reduce && (a.num_chunks >= kWideRows || near)) {
        const size_t blocks = (a.n + kWideTargets - 1) / kWideTargets;
        const size_t cap = static_cast<size_t>(sm_count > 0 ? sm_count : 148) * 8;
        const unsigned grid = static_cast<unsigned>(blocks < 1 ? 1 : (blocks < cap ? blocks : cap));
        if (near)
            return launch_pdl(stage_kernel<MODE, true, true>, dim3(grid), dim3(256), 0, stream, a);
        return launch_pdl(stage_kernel<MODE, true>, dim3(grid), dim3(256), 0, stream, a);
    }
    return launch_pdl(stage_kernel<MODE, false>, dim3(grid_for(a.n, sm_count)), dim3(256), 0,
                      stream, a);
}

cudaError_t launch_stage(const StageArgs &a, cudaStream_t stream, int sm_count) {
    switch (a.mode) {
    case STAGE_REDUCE_ONLY:
        return launch_stage_mode<STAGE_REDUCE_ONLY>(a, stream, sm_count);
    case STAGE_POSITION:
        return launch_stage_mode<STAGE_POSITION>(a, stream, sm_count);
    case STAGE_RK4_COMBINE:
        return launch_stage_mode<STAGE_RK4_COMBINE>(a, stream, sm_count);
    case STAGE_DOPRI_ERROR:
        return launch_stage_mode<STAGE_DOPRI_ERROR>(a, stream, sm_count);
    default:
        return cudaErrorInvalidValue;
    }
}

// ---------------------------------------------------------------------------------------------
// Whole steps of a small FP64 population in one cooperative launch: RK4 steps, or one adaptive DOPRI5
// step with its rejected attempts. Below N ~ 2000 a step's launches (9 for RK4, 13 an attempt) take
// longer to schedule than to run, so one CTA per SM keeps the whole loop: each CTA owns a range of
// targets, and a grid barrier separates the evaluations.
//
// The results are bit for bit those of the launch sequence: a target's velocity is summed chunk by
// chunk (the ordered kernel's chunks, sources in index order, pair<true> with the self flag), the
// chunk sums are added as sum_chunks adds them, and the stage arithmetic is the stage kernel's.
//
// What bounds it is latency. One stage of N = 1024 in the plane: the barrier (arrival and poll, each a
// round trip to L2), the load of all positions into shared memory, the chunk sums (up to 31 chunks,
// so that 217 threads of an SM have one; their sources unrolled, so that the pairs' chains overlap)
// and the finish, whose inputs -- the step's start and the earlier stage velocities -- stay in
// shared memory: 0.9, 2.9, 1.5 and 2.4 thousand cycles for load, sums, finish and barrier. Measured
// against the previous kernel (RK4, us a step: 128 threads' worth of chunks, positions and inputs
// reloaded in the finish, a fenced atomic and a status read a barrier): plane N = 64 20 -> 14, 1024
// 33 -> 17, 2047 47 -> 33; disk 2048 87 -> 52; box 1024 130 -> 31 (with ZetaPair). DOPRI5 against the
// captured graph of launches (us a step, host included): disk 301 85 -> 57, plane 1024 81 -> 58, box
// 1024 192 -> 83.

// Grid barrier over the CTAs of a cooperative launch. The arrival counter starts at zero (the control
// block is reset before the launch): the r-th barrier is open once it has counted r * gridDim.x
// (pv_barrier.cuh lays the word out). One release-add per CTA, then polling with acquire loads.
//
// A CTA that met an error in the phase adds it to its arrival, in one of two fields by the barrier's
// parity; every CTA that passes the barrier sees it there and stops. (A CTA can be one barrier ahead
// of a slow poller, never two, so the poller's own field holds its own barrier's errors only.)
//
// A wait that outlasts `limit` polls breaks the barrier instead of walking away from it: a
// compare-and-swap sets the broken flag of the barrier's parity in the counter, and succeeds only if
// the counter has not moved since it was read. Every CTA therefore agrees on each barrier: either it
// opened (the last arrival came before the swap) and all pass it -- also a slow poller that finds
// the next one broken -- or it is broken and none does: later arrivals and pollers see the flag and
// return. The breaker sets ST_TIMEOUT. Since the state is written only in phases that follow an
// open barrier, a timeout leaves it at the last completed step.
struct GridBarrier {
    unsigned long long *arrivals;
    int *status;
    uint32_t limit;
    unsigned long long open_at;  // of the next barrier
    unsigned parity;

    __device__ __forceinline__ explicit GridBarrier(const SmallSteps &p)
        : arrivals(&p.ctl->arrivals), status(&p.ctl->status), limit(p.spin_limit), open_at(0ull),
          parity(0u) {}

    // Returns true when the barrier opened and no CTA arrived with an error. bad: this thread met one.
    __device__ __forceinline__ bool wait(bool bad) {
        __shared__ int go;
        const int any_bad = __syncthreads_or(bad);
        open_at += barrier::arrivals(gridDim.x);
        parity ^= 1u;
        if (threadIdx.x == 0) {
            const unsigned long long broken = barrier::broken(parity);
            const unsigned long long mine = barrier::arrival(any_bad != 0, parity);
            // this CTA's writes, ordered by the __syncthreads, before its arrival
            asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(arrivals), "l"(mine)
                         : "memory");
            unsigned long long now;
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(now) : "l"(arrivals) : "memory");
            int ok = 1;
            for (uint32_t it = 0;;) {
                if (now & broken) {
                    ok = 0;
                    break;
                }
                if (barrier::open(now, open_at))
                    break;
                if (it >= limit) {
                    const unsigned long long seen = atomicCAS(arrivals, now, now | broken);
                    if (seen == now) {
                        set_status(status, ST_TIMEOUT);
                        ok = 0;
                        break;
                    }
                    now = seen;  // another CTA arrived (or broke it) meanwhile: look again
                    continue;
                }
                ++it;
                if (it > 256)
                    __nanosleep(32);
                asm volatile("ld.acquire.gpu.global.u64 %0, [%1];"
                             : "=l"(now)
                             : "l"(arrivals)
                             : "memory");
            }
            if (ok && barrier::errors(now, parity))
                ok = 0;
            go = ok;
        }
        __syncthreads();
        return go != 0;
    }
};

// The same steps in one cluster of kClusterSteps CTAs, for populations whose pairs so few SMs evaluate
// as fast as the grid exchanges positions: the barrier is the hardware's, and each stage's positions go
// straight into the other buffer of every CTA's shared memory, where the next evaluation reads them. A
// CTA that met an error tells every CTA through a flag there, by the barrier's parity as above. The
// hardware's barrier has no limit to set; it cannot stay shut, since a cluster's CTAs are resident
// together and each takes the same way through the phases. A stage saves about 1 us: RK4 steps at
// N = 128, grid and cluster: plane 12.1 and 8.2 us, disk 14.1 and 10.1, box 18.2 and 14.2.
constexpr unsigned kClusterSteps = 16;

__device__ __forceinline__ uint32_t remote_shared(const void *local, unsigned rank) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;"
        : "=r"(a)
        : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(local))), "r"(rank));
    return a;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

struct ClusterBarrier {
    int *flags;  // [2] in this CTA's shared memory
    unsigned parity;

    __device__ __forceinline__ explicit ClusterBarrier(const SmallSteps &) : parity(0u) {
        __shared__ int shared_flags[2];
        flags = shared_flags;
        if (threadIdx.x < 2)
            flags[threadIdx.x] = 0;
    }
    __device__ __forceinline__ bool wait(bool bad) {
        parity ^= 1u;
        if (bad)
            for (unsigned rank = 0; rank < kClusterSteps; ++rank)
                asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(
                                 remote_shared(flags + parity, rank)),
                             "r"(1)
                             : "memory");
        cluster_sync();
        return *static_cast<volatile int *>(flags + parity) == 0;
    }
};

// Sources whose pair chains overlap in a thread's chunk sum.
template <class Pair> struct ChunkUnroll { static constexpr int value = 4; };
template <> struct ChunkUnroll<InfinitePair> { static constexpr int value = 16; };
template <> struct ChunkUnroll<DiskPair> { static constexpr int value = 8; };

constexpr int kStepThreads = 256;

// Shared memory of a CTA: all sources, its targets' chunk sums, and per target what its finish
// keeps from stage to stage.
template <bool CLUSTER> struct StepShared {
    double *x, *y, *g;    // [n]
    double *xn, *yn;      // [n]: a cluster's next positions
    double *qu, *qv;      // [targets][chunks]
    double *k;            // [7][2][targets]: stage velocities
    double *x0, *y0;      // [targets]: the step's start
    __device__ __forceinline__ StepShared(double *base, size_t n, size_t targets, int chunks) {
        const size_t np = (n + 1) & ~static_cast<size_t>(1);
        x = base;
        y = x + np;
        g = y + np;
        qu = g + np;
        qv = qu + targets * chunks;
        k = qv + targets * chunks;
        x0 = k + 14 * targets;
        y0 = x0 + targets;
        xn = y0 + targets;
        yn = xn + np;
    }
    // Position of target i for the next evaluation: to every CTA, or to the exchange's buffer `to`.
    __device__ __forceinline__ void publish(const SmallSteps &p, int to, size_t i, double px,
                                            double py) const {
        if (CLUSTER) {
#pragma unroll 4
            for (unsigned rank = 0; rank < kClusterSteps; ++rank) {
                asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(remote_shared(xn + i, rank)),
                             "d"(px)
                             : "memory");
                asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(remote_shared(yn + i, rank)),
                             "d"(py)
                             : "memory");
            }
        } else {
            p.px[to][i] = px;
            p.py[to][i] = py;
        }
    }
    // After the barrier that follows publish().
    __device__ __forceinline__ void turn() {
        if (CLUSTER) {
            double *t = x;
            x = xn;
            xn = t;
            t = y;
            y = yn;
            yn = t;
        }
    }
    // A cluster's first positions, and every CTA started before any writes into another's memory.
    __device__ __forceinline__ void begin(const SmallSteps &p) const {
        if (CLUSTER) {
            for (size_t j = threadIdx.x; j < p.n; j += kStepThreads) {
                x[j] = p.x[j];
                y[j] = p.y[j];
            }
            cluster_sync();
        }
    }
};
constexpr size_t step_shared_bytes(size_t n, size_t targets, size_t units, bool cluster) {
    const size_t np = (n + 1) & ~static_cast<size_t>(1);
    return ((cluster ? 5 : 3) * np + 2 * units + 16 * targets) * sizeof(double);
}
// The most that small_steps_eligible() and small_steps_in_cluster() let a launch ask for.
constexpr size_t step_shared_max(bool cluster) {
    return cluster ? step_shared_bytes(kSmallStepsMaxN, (kSmallStepsMaxN + kClusterSteps - 1) / kClusterSteps,
                                       kStepThreads, true)
                   : step_shared_bytes(kSmallStepsMaxN, kStepThreads, kStepThreads * (kWideRows - 1), false);
}
static_assert(step_shared_max(false) <= 226 * 1024 && step_shared_max(true) <= 226 * 1024,
              "a CTA's shared memory, with 1 KB to spare for the kernels' own");

// One evaluation: positions (px, py) into shared memory (a cluster's are there), then the chunk sums of
// the CTA's targets [t0, t0 + mine).
template <class Pair, bool CLUSTER>
__device__ __forceinline__ void step_evaluate(const SmallSteps &p, const StepShared<CLUSTER> &sh,
                                              const double *px, const double *py, size_t t0,
                                              int mine) {
    if (!CLUSTER) {
        const int n2 = static_cast<int>(p.n / 2);
        const double2 *px2 = reinterpret_cast<const double2 *>(px);
        const double2 *py2 = reinterpret_cast<const double2 *>(py);
#pragma unroll 4  // the loads of several iterations in flight at once
        for (int j = threadIdx.x; j < n2; j += kStepThreads) {
            reinterpret_cast<double2 *>(sh.x)[j] = __ldcg(px2 + j);
            reinterpret_cast<double2 *>(sh.y)[j] = __ldcg(py2 + j);
        }
        if ((p.n & 1) && threadIdx.x == 0) {
            sh.x[p.n - 1] = __ldcg(px + p.n - 1);
            sh.y[p.n - 1] = __ldcg(py + p.n - 1);
        }
        __syncthreads();
    }
    const int nc = p.num_chunks;
    for (int w = threadIdx.x; w < mine * nc; w += kStepThreads) {
        const int li = w % mine, c = w / mine;
        const int i = static_cast<int>(t0) + li;
        const int j0 = c * p.chunk, j1 = min(j0 + p.chunk, static_cast<int>(p.n));
        const double tx = sh.x[i], ty = sh.y[i];
        double u = 0.0, v = 0.0;
        // unrolled so that the independent work of several sources overlaps; the sums still take
        // the sources in index order
        constexpr int kUnroll = ChunkUnroll<Pair>::value;
        int j = j0;
        for (; j + kUnroll <= j1; j += kUnroll) {
#pragma unroll
            for (int q = 0; q < kUnroll; ++q)
                Pair::template pair<true>(p.g, tx, ty, sh.x[j + q], sh.y[j + q], sh.g[j + q],
                                          i == j + q, u, v);
        }
#pragma unroll 2
        for (; j < j1; ++j)
            Pair::template pair<true>(p.g, tx, ty, sh.x[j], sh.y[j], sh.g[j], i == j, u, v);
        sh.qu[li * nc + c] = u;
        sh.qv[li * nc + c] = v;
    }
    __syncthreads();
}

// The velocity of target li from its chunk sums (the slow path included), kept as stage s's. Returns
// an error status, or 0.
template <bool CLUSTER>
__device__ __forceinline__ int step_velocity(const SmallSteps &p, const StepShared<CLUSTER> &sh,
                                             int li, size_t i, int targets, int s) {
    double ku, kv;
    const double *qu = sh.qu + li * p.num_chunks, *qv = sh.qv + li * p.num_chunks;
    sum_chunks(
        p.num_chunks,
        [&](int c, double &ru, double &rv) {
            ru = qu[c];
            rv = qv[c];
        },
        ku, kv);
    int verdict = 0;
    if (!isfinite(ku) || !isfinite(kv))  // recomputed from this phase's positions
        verdict = slow_target(p.g, sh.x, sh.y, p.gamma, p.n, i, ku, kv);
    sh.k[(2 * s) * targets + li] = ku;
    sh.k[(2 * s + 1) * targets + li] = kv;
    return verdict;
}

// Stage position x0 + dt sum_j a_j k_j of component `part` (makeStage, src/timestep.cpp:19-30).
template <bool CLUSTER>
__device__ __forceinline__ double step_position(const StepShared<CLUSTER> &sh, const double *row,
                                                int ncoef, int part, int li, int targets, double x0,
                                                double dt) {
    double d = 0.0;
    for (int j = 0; j < ncoef; ++j)
        if (row[j] != 0.0)
            d = __dadd_rn(d, __dmul_rn(row[j], sh.k[(2 * j + part) * targets + li]));
    return __dadd_rn(x0, __dmul_rn(dt, d));
}

template <class Pair, bool CLUSTER>
__global__ void __launch_bounds__(kStepThreads, 1) rk4_steps_kernel(const SmallSteps p) {
    extern __shared__ __align__(16) double smem[];
    const int targets = static_cast<int>((p.n + gridDim.x - 1) / gridDim.x);
    const size_t t0 = static_cast<size_t>(blockIdx.x) * targets;
    const int mine = t0 < p.n ? static_cast<int>(min(static_cast<size_t>(targets), p.n - t0)) : 0;
    StepShared<CLUSTER> sh(smem, p.n, targets, p.num_chunks);
    for (size_t j = threadIdx.x; j < p.n; j += kStepThreads)
        sh.g[j] = p.gs[j];
    std::conditional_t<CLUSTER, ClusterBarrier, GridBarrier> barrier(p);
    sh.begin(p);
    const int li = threadIdx.x;  // a target's finish is its own thread's
    const size_t i = t0 + li;
    for (uint64_t step = 0; step < p.steps; ++step) {
        for (int s = 0; s < 4; ++s) {
            // evaluation point: the state, or for a step's first stage after the first step the
            // previous step's combination (not yet copied into the state); then the last stage's
            const double *px = s == 0 ? (step > 0 ? p.px[1] : p.x) : p.px[(s - 1) & 1];
            const double *py = s == 0 ? (step > 0 ? p.py[1] : p.y) : p.py[(s - 1) & 1];
            step_evaluate<Pair, CLUSTER>(p, sh, px, py, t0, mine);
            int error = 0;
            if (li < mine) {
                if (s == 0) {
                    sh.x0[li] = sh.x[i];
                    sh.y0[li] = sh.y[i];
                    if (step > 0) {  // the accept of the previous step
                        p.x[i] = sh.x[i];
                        p.y[i] = sh.y[i];
                    }
                }
                error = step_velocity(p, sh, li, i, targets, s);
                double nx, ny;
                if (s < 3) {
                    nx = step_position(sh, p.rows[s + 1], s + 1, 0, li, targets, sh.x0[li], p.dt);
                    ny = step_position(sh, p.rows[s + 1], s + 1, 1, li, targets, sh.y0[li], p.dt);
                    error = max(error, position_error(p.g, nx, ny));
                } else {
                    const double *k = sh.k + li;
                    nx = rk4_point(sh.x0[li], p.dt, k[0], k[2 * targets], k[4 * targets],
                                   k[6 * targets]);
                    ny = rk4_point(sh.y0[li], p.dt, k[targets], k[3 * targets], k[5 * targets],
                                   k[7 * targets]);
                    if (!isfinite(nx) || !isfinite(ny))
                        error = max(error, static_cast<int>(ST_NONFINITE_POSITION));
                }
                sh.publish(p, s & 1, i, nx, ny);
                if (error)
                    set_status(&p.ctl->status, error);
            }
            if (!barrier.wait(error != 0))
                return;
            sh.turn();
        }
    }
    if (li < mine) {  // the last step's accept
        p.x[i] = CLUSTER ? sh.x[i] : __ldcg(p.px[1] + i);
        p.y[i] = CLUSTER ? sh.y[i] : __ldcg(p.py[1] + i);
    }
}

// One adaptive step (src/timestep.cpp:62-120). need_k0: the derivative at the state is not cached in
// (k0x, k0y). A rejected attempt changes only the step size, so the next one starts from the same
// k0 without leaving the kernel; an accepted one updates the state and k0.
template <class Pair, bool CLUSTER>
__global__ void __launch_bounds__(kStepThreads, 1) dopri_step_kernel(const SmallSteps p) {
    extern __shared__ __align__(16) double smem[];
    __shared__ double s_error;
    const int targets = static_cast<int>((p.n + gridDim.x - 1) / gridDim.x);
    const size_t t0 = static_cast<size_t>(blockIdx.x) * targets;
    const int mine = t0 < p.n ? static_cast<int>(min(static_cast<size_t>(targets), p.n - t0)) : 0;
    StepShared<CLUSTER> sh(smem, p.n, targets, p.num_chunks);
    for (size_t j = threadIdx.x; j < p.n; j += kStepThreads)
        sh.g[j] = p.gs[j];
    std::conditional_t<CLUSTER, ClusterBarrier, GridBarrier> barrier(p);
    sh.begin(p);
    const int li = threadIdx.x;
    const size_t i = t0 + li;
    const bool owner = li < mine;
    DeviceControl *ctl = p.ctl;
    const double minimum = ctl->minimum_time_step, maximum = ctl->maximum_time_step;
    double dt = ctl->dt;
    unsigned rejected = 0;
    if (owner) {
        sh.x0[li] = p.x[i];
        sh.y0[li] = p.y[i];
        if (!p.need_k0) {
            sh.k[li] = p.k0x[i];
            sh.k[targets + li] = p.k0y[i];
        }
    }
    for (int attempt = 0;; ++attempt) {
        // the error words alternate; this attempt's was last read two attempts ago
        unsigned long long *word = attempt & 1 ? &ctl->err_bits2 : &ctl->err_bits;
        if (attempt > 0 && blockIdx.x == 0 && threadIdx.x == 0)
            *word = 0ull;
        double x5 = 0.0, y5 = 0.0, local = 0.0;
        for (int s = 0; s < 7; ++s) {
            const bool evaluate = s > 0 || (p.need_k0 && attempt == 0);
            if (evaluate)
                step_evaluate<Pair, CLUSTER>(p, sh, s == 0 ? p.x : p.px[(s - 1) & 1],
                                             s == 0 ? p.y : p.py[(s - 1) & 1], t0, mine);
            int error = 0;
            if (owner) {
                if (evaluate)
                    error = step_velocity(p, sh, li, i, targets, s);
                if (s < 6) {
                    x5 = step_position(sh, p.rows[s + 1], s + 1, 0, li, targets, sh.x0[li], dt);
                    y5 = step_position(sh, p.rows[s + 1], s + 1, 1, li, targets, sh.y0[li], dt);
                    sh.publish(p, s & 1, i, x5, y5);
                    error = max(error, position_error(p.g, x5, y5));
                } else {  // (x5, y5): the fifth-order point, the position of k6
                    double xe = 0.0, ye = 0.0;
                    for (int j = 0; j < 7; ++j) {
                        if (p.w[j] == 0.0)
                            continue;
                        const double h = __dmul_rn(dt, p.w[j]);
                        xe = __dadd_rn(xe, __dmul_rn(h, sh.k[(2 * j) * targets + li]));
                        ye = __dadd_rn(ye, __dmul_rn(h, sh.k[(2 * j + 1) * targets + li]));
                    }
                    const double xs = error_scale(ctl, sh.x0[li], x5);
                    const double ys = error_scale(ctl, sh.y0[li], y5);
                    if (!isfinite(xe) || !isfinite(ye) || !isfinite(xs) || !isfinite(ys) ||
                        !(xs > 0.0) || !(ys > 0.0))
                        error = max(error, static_cast<int>(ST_DOPRI_NONFINITE));
                    else
                        local = max_ref(__ddiv_rn(fabs(xe), xs), __ddiv_rn(fabs(ye), ys));
                }
                if (error)
                    set_status(&ctl->status, error);
            }
            if (s == 6 && threadIdx.x < 32 * ((mine + 31) / 32)) {  // whole warps of owners
                for (int off = 16; off > 0; off >>= 1)
                    local = max_ref(local, __shfl_xor_sync(0xffffffffu, local, off));
                if ((threadIdx.x & 31) == 0)
                    atomicMax(word, ordered_bits(local));
            }
            if (!barrier.wait(error != 0)) {
                if (blockIdx.x == 0 && threadIdx.x == 0)
                    ctl->attempts = attempt + 1;
                return;
            }
            if (s < 6)
                sh.turn();
        }
        if (threadIdx.x == 0)
            s_error = __longlong_as_double(
                static_cast<long long>(*reinterpret_cast<volatile unsigned long long *>(word)));
        __syncthreads();
        // every thread takes the same decision from the same numbers
        const double error = s_error;
        int accepted;
        double suggested, next_dt;
        const int failed =
            dopri_decide(error, dt, minimum, maximum, rejected, accepted, suggested, next_dt);
        if (accepted && owner) {
            p.x[i] = x5;
            p.y[i] = y5;
            p.k0x[i] = sh.k[12 * targets + li];
            p.k0y[i] = sh.k[13 * targets + li];
        }
        if ((accepted || failed) && blockIdx.x == 0 && threadIdx.x == 0) {
            ctl->accepted = accepted;
            ctl->rejected = rejected;
            ctl->attempts = attempt + 1;
            if (accepted)
                store_accepted(ctl, dt, suggested, error, rejected);
            else
                set_status(&ctl->status, failed);
        }
        if (accepted || failed)
            return;
        dt = next_dt;
    }
}

// While a CTA of the cluster has a thread for each (target, chunk); the box, whose pairs take five times
// the plane's FP64 cycles, while it has two. Measured at both sides (us an RK4 step, cluster and grid):
// plane N = 300 11.4 and 14.1, 400 17.8 and 13.4; disk 300 14.8 and 15.4, 400 23.8 and 14.6; box 200
// 14.8 and 18.4, 256 20.9 and 18.5.
bool small_steps_in_cluster(const GeometryConsts &g, size_t n, int num_chunks) {
    const size_t units = (n + kClusterSteps - 1) / kClusterSteps * static_cast<size_t>(num_chunks);
    return units <= (g.geometry == GEO_PERIODIC ? kStepThreads / 2 : kStepThreads);
}

bool small_steps_eligible(size_t n, int num_chunks, int sm_count) {
    const size_t grid = static_cast<size_t>(sm_count > 0 ? sm_count : 148);
    return n >= 1 && n <= kSmallStepsMaxN && num_chunks >= 1 && num_chunks < kWideRows &&
           grid <= barrier::kMaxCtas && (n + grid - 1) / grid <= kStepThreads;
}

namespace {
// The whole grid, one CTA per SM, cooperative (every CTA resident, or no launch at all), or one cluster.
// The kernel's limit of shared memory belongs to the function, which the contexts of all host threads
// launch: each sets it to the same value, the most any of them needs, since one that set its own launch's
// size would take it from under another's.
template <class Kernel>
cudaError_t launch_steps(Kernel kernel, const SmallSteps &p, size_t grid, bool cluster,
                         cudaStream_t stream) {
    const size_t targets = (p.n + grid - 1) / grid;
    const size_t smem = step_shared_bytes(p.n, targets, targets * p.num_chunks, cluster);
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(step_shared_max(cluster)));
    if (e == cudaSuccess && cluster)
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess)
        return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(grid));
    cfg.blockDim = dim3(kStepThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    if (cluster) {
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = kClusterSteps;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    } else {
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, p);
}

template <class Pair>
cudaError_t launch_small(const SmallSteps &p, int sm_count, cudaStream_t stream) {
    if (p.cluster) {
        const cudaError_t e =
            p.dopri ? launch_steps(dopri_step_kernel<Pair, true>, p, kClusterSteps, true, stream)
                    : launch_steps(rk4_steps_kernel<Pair, true>, p, kClusterSteps, true, stream);
        if (e == cudaSuccess)
            return e;
        cudaGetLastError();  // no GPC with that many SMs free for a cluster: the grid
    }
    const size_t grid =
        std::min<size_t>(static_cast<size_t>(sm_count > 0 ? sm_count : 148), p.n);
    return p.dopri ? launch_steps(dopri_step_kernel<Pair, false>, p, grid, false, stream)
                   : launch_steps(rk4_steps_kernel<Pair, false>, p, grid, false, stream);
}
} // namespace

cudaError_t launch_small_steps(const SmallSteps &p, int sm_count, cudaStream_t stream) {
    if (!small_steps_eligible(p.n, p.num_chunks, sm_count) || (!p.dopri && p.steps == 0))
        return cudaErrorInvalidValue;
    switch (p.g.geometry) {
    case GEO_INFINITE:
        return launch_small<InfinitePair>(p, sm_count, stream);
    case GEO_PERIODIC:
        return p.g.zeta ? launch_small<ZetaPair>(p, sm_count, stream)
                        : launch_small<PeriodicPair>(p, sm_count, stream);
    case GEO_DISK:
        return launch_small<DiskPair>(p, sm_count, stream);
    default:
        return cudaErrorInvalidValue;
    }
}

cudaError_t launch_accept(double *x, double *y, const double *xt, const double *yt, double *k0x,
                          double *k0y, const double *k6x, const double *k6y, size_t n, int dopri,
                          DeviceControl *ctl, cudaStream_t stream) {
    return launch_pdl(accept_kernel, dim3(grid_for(n, 0)), dim3(256), 0, stream, x, y, xt, yt, k0x,
                      k0y, k6x, k6y, n, dopri, ctl);
}

} // namespace pvb
