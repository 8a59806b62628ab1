/*
 * mfcfd_kernels.cu - the FP64 q-LSKUM iteration on sm_100a.
 *
 * One iteration (fpi_solver.f90:27-36) is this launch sequence:
 *   k_qderiv      q_derivatives + timestep_delt     thread per point
 *   k_flux        eval_flux_residual                warp per point; with the
 *                 chain schedule also what follows, otherwise:
 *   k_pending     sweep hand-off words set to "not yet published"
 *   k_dinv_gold   D_inv, fluxes of prim in the shared interior frame,
 *                 flux increments of points the sweeps do not update
 *   k_sweep_chain x2  forward / backward LU-SGS sweep: static chains walked
 *                 by teams of warps on all SMs, mfcfd_chain.cuh
 *                 (k_sweep_df: dynamic topological order;
 *                 k_sweep_levels: one CTA, level by level)
 *   k_update      state_update_implicit + next iteration's U and q
 *                 (k_update_ss: supersonic points' copies, in order)
 *   k_reduce_*    res_new (deterministic two-pass sum)
 * State stays resident in HBM in the reference's point-major layout.
 *
 * Built with -fmad=false: every multiply and add rounds separately, as in
 * the reference's build; see mfcfd_physics.cuh for the expression order.
 */
#include <cuda_runtime.h>

#include <mutex>
#include <type_traits>
#include <utility>
#include <string>

#include "mfcfd_internal.h"
#include "mfcfd_physics.cuh"
#include "mfcfd_publish.cuh"

namespace mfcfd {

constexpr int FLUX_WARPS = 4;            // warps per CTA in k_flux
constexpr int FLUX_SMEM_PER_WARP = NDIR * MAX_SLOTS * 5 + MAX_SLOTS * 3;   // doubles
constexpr int SWEEP_THREADS = 512;
constexpr int SWEEP_WARPS = SWEEP_THREADS / 32;
constexpr int RED_THREADS = 256;
constexpr unsigned FULL = 0xffffffffu;

// ---------------------------------------------------------------- U and q

// The speed of timestep_delt.f90:243-247 at a point: |u| + 3 sqrt(p / rho).
__device__ __forceinline__ double signal_speed(const double p[5]) {
    const double mod_u = sqrt(p[1] * p[1] + p[2] * p[2] + p[3] * p[3]);
    return mod_u + 3.0 * sqrt(p[4] / p[0]);
}

// compute_conserved_vector + eval_q_variables for every point.
__global__ void k_conserved_q(DevCloud d) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.n) return;
    Frame F;
    load_frame(d.frame + 9 * (size_t)i, F);
    double p[5], U[5], q[5];
#pragma unroll
    for (int r = 0; r < 5; ++r) p[r] = d.prim[5 * (size_t)i + r];
    primitive_to_rotated_conserved(p, F, U);
    primitive_to_q(p, q);
    d.pos[4 * (size_t)i + 3] = signal_speed(p);
#pragma unroll
    for (int r = 0; r < 5; ++r) {
        d.U[5 * (size_t)i + r] = U[r];
        d.q[5 * (size_t)i + r] = q[r];
    }
}

// ---------------------------------------------------------------- q-derivatives

// One inner iteration of the second-order q-derivatives
// (q_derivatives.f90:116-201): least squares over conn of the differences of
// the half-step reconstructions q - dq.del/2 at both ends, from dq_in into
// dq_out (the reference's point%temp, copied back after the pass).
__global__ void __launch_bounds__(128) k_qinner(DevCloud d, const double *dq_in, double *dq_out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.n) return;
    const double xi = d.x[i], yi = d.y[i], zi = d.z[i];
    double qi[5], dqi[15];
#pragma unroll
    for (int r = 0; r < 5; ++r) qi[r] = d.q[5 * (size_t)i + r];
#pragma unroll
    for (int c = 0; c < 15; ++c) dqi[c] = dq_in[15 * (size_t)i + c];
    double xx = 0, yy = 0, zz = 0, xy = 0, yz = 0, zx = 0;
    double sx[5] = {0, 0, 0, 0, 0}, sy[5] = {0, 0, 0, 0, 0}, sz[5] = {0, 0, 0, 0, 0};
    const int nb = d.nbhs[i];
    const int32_t *cn = d.conn + (size_t)MAX_CONN * i;
    for (int j = 0; j < nb; ++j) {
        const int k = cn[j];
        const double delx = d.x[k] - xi, dely = d.y[k] - yi, delz = d.z[k] - zi;
        const double w = d.wq ? d.wq[(size_t)MAX_CONN * i + j] : 1.0;
        xx = xx + delx * delx * w;
        yy = yy + dely * dely * w;
        zz = zz + delz * delz * w;
        xy = xy + delx * dely * w;
        yz = yz + dely * delz * w;
        zx = zx + delz * delx * w;
        const double *dqk = dq_in + 15 * (size_t)k;
#pragma unroll
        for (int r = 0; r < 5; ++r) {
            const double qti = qi[r] - 0.5 * (delx * dqi[3 * r] + dely * dqi[3 * r + 1] + delz * dqi[3 * r + 2]);
            const double qtn = d.q[5 * (size_t)k + r] - 0.5 * (delx * dqk[3 * r] + dely * dqk[3 * r + 1] + delz * dqk[3 * r + 2]);
            const double t = qtn - qti;
            sx[r] = sx[r] + w * delx * t;
            sy[r] = sy[r] + w * dely * t;
            sz[r] = sz[r] + w * delz * t;
        }
    }
    const double g[6] = {xx, yy, zz, xy, yz, zx};
    const double det = xx * (yy * zz - yz * yz) - xy * (xy * zz - yz * zx) + zx * (xy * yz - yy * zx);
    const double one_by_det = 1.0 / det;
#pragma unroll
    for (int r = 0; r < 5; ++r) {
        dq_out[15 * (size_t)i + 3 * r + 0] = cramer_num(0, g, sx[r], sy[r], sz[r]) * one_by_det;
        dq_out[15 * (size_t)i + 3 * r + 1] = cramer_num(1, g, sx[r], sy[r], sz[r]) * one_by_det;
        dq_out[15 * (size_t)i + 3 * r + 2] = cramer_num(2, g, sx[r], sy[r], sz[r]) * one_by_det;
    }
}

// ---------------------------------------------------------------- hand-off words

// Hand-off of increments between warps.  Before the sweeps, k_dinv_gold sets
// dUp, dUn, dgf and dgb of every swept point to DU_PENDING, a signalling-NaN
// bit pattern that no arithmetic result has (arithmetic NaNs are quiet).  A
// producer stores its values with strong (relaxed, gpu-scope) 8-byte stores;
// a consumer polls the 8-byte words it needs with strong loads until none is
// DU_PENDING.  Each word is single-copy atomic, so a value read that is not
// DU_PENDING is the final one: no flags and no fences are needed.
constexpr unsigned long long DU_PENDING = 0xFFF4DEADBEEF0001ull;

__device__ __forceinline__ unsigned long long ld_relaxed_b64(const double *p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void ld_relaxed_v2(const double *p, unsigned long long &a, unsigned long long &b) {
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ void st_relaxed_f64(double *p, double v) {
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}

// Polls give up after SPIN_LIMIT rounds (about a second; d.spin_limit when
// set), or soon after another lane gave up: the failure goes to *d.err (the
// host reports MFCFD_ERR_TIMEOUT and the iteration's results are invalid).
constexpr int SPIN_LIMIT = 1 << 21;

__device__ __forceinline__ bool spin_continue(int &it, const DevCloud &d) {
    ++it;
    if ((it & 1023) == 0) {
        if (*(volatile int *)d.err) return false;
        __nanosleep(64);
    }
    if (it > (d.spin_limit > 0 ? d.spin_limit : SPIN_LIMIT)) {
        atomicExch(d.err, 1);
        return false;
    }
    return true;
}

__device__ __forceinline__ bool is_pending(double v) {
    return (unsigned long long)__double_as_longlong(v) == DU_PENDING;
}

// Poll one word until it is published.
__device__ __forceinline__ double poll_word(const double *p, const DevCloud &d) {
    unsigned long long v;
    int spins = 0;
    do {
        v = ld_relaxed_b64(p);
    } while (v == DU_PENDING && spin_continue(spins, d));
    return __longlong_as_double((long long)v);
}

__device__ __forceinline__ bool ready5(const unsigned long long v[5]) {
    return v[0] != DU_PENDING && v[1] != DU_PENDING && v[2] != DU_PENDING && v[3] != DU_PENDING &&
           v[4] != DU_PENDING;
}

// ---------------------------------------------------------------- flux residual

// Limited midpoint reconstruction of point j's q toward the offset
// (delx, dely, delz), then q -> primitive (interior_flux_dGxpos.f90:92-96,
// limiters.f90:12-52, qvariables_to_primitive_variables.f90:9-31).
template <typename R>
__device__ __forceinline__ void reconstruct(const DevCloud &d, int j, R delx, R dely, R delz, R prim[5]) {
    const double *qj = d.q + 5 * (size_t)j;
    const double *dqj = d.dq + 15 * (size_t)j;
    const double *qmj = d.qm + 10 * (size_t)j;
    const R eps2 = (R)d.eps2[j];
    R qt[5];
#pragma unroll
    for (int r = 0; r < 5; ++r) {
        const R q = (R)qj[r];
        const R temp = delx * (R)dqj[3 * r] + dely * (R)dqj[3 * r + 1] + delz * (R)dqj[3 * r + 2];
        const R del_neg = (q - R(0.5) * temp) - q;
        R phi = R(1.0);
        if (!(r_abs(del_neg) <= R(MF_LIM_EPS))) {
            const R del_pos = del_neg > R(0.0) ? (R)qmj[2 * r] - q : (R)qmj[2 * r + 1] - q;
            R num = (del_pos * del_pos) + eps2;
            num = num * del_neg + R(2.0) * del_neg * del_neg * del_pos;
            R den = del_pos * del_pos + R(2.0) * del_neg * del_neg;
            den = den + del_neg * del_pos + eps2;
            den = den * del_neg;
            const R t = num / den;
            phi = (t < R(1.0)) ? t : R(1.0);
        }
        qt[r] = q - R(0.5) * phi * temp;
    }
    qtilde_to_primitive(qt, prim);
}

// Per-list diagonal terms of D_inv (implicit_D_inv_interior.f90:46-417 /
// implicit_D_inv_wall.f90:45-356 with the geometry-only sums precomputed).
// u: the velocity component of list dd's axis; as: the speed of sound;
// row: the geometry row (dd, or 5 for an outer point's z+ over conn).
__device__ __forceinline__ double dinv_term(const DevCloud &d, int i, int dd, double u, double as, int row) {
    const double *g = d.geo + (size_t)i * GEO_STRIDE + (row - dd) * 8;
    const double temp = g[dd * 8 + G_DNUM], det = g[dd * 8 + G_DET];
    if ((dd & 1) == 0) {
        const double t1 = u + as;
        return 0.50 * fabs(t1 + fabs(t1)) * temp / det;
    }
    const double t1 = u - as;
    return -(0.50 * fabs(t1 - fabs(t1)) * temp / det);
}

__device__ __forceinline__ double dinv_term(const DevCloud &d, int i, int dd, double u, double as) {
    return dinv_term(d, i, dd, u, as, dd);
}

// implicit_D_inv_outer.f90:17-363 (backup driver) from the terms of rows
// 0-3 and of row 5 (z+ over conn): no minus on the x-/y- terms, the source's
// order of operations, and 1/delt of the tangential offset the direction
// loops leave behind (outer_delt; NaN: the time step).
__device__ __forceinline__ double dinv_outer(const DevCloud &d, int i, const double g5[5]) {
    double dt = d.outer_delt[i];
    if (dt != dt) dt = d.delt[i];
    const double temp = (1.0 / dt) - g5[0] + (-g5[1]) - g5[2] + (-g5[3]) - g5[4];
    return 1.0 / temp;
}

__device__ __forceinline__ double dinv_combine(int cls, double delt, const double gd[NDIR]) {
    double temp;
    if (cls == CLS_WALL) temp = (1.0 / delt) - 2.0 * (gd[0] + gd[1] + gd[2] + gd[3] + gd[5]);
    else temp = (1.0 / delt) - (gd[0] + gd[1] + gd[2] + gd[3] + gd[4] + gd[5]);
    return 1.0 / temp;
}

// The sweep inputs of point i (chain schedule; as k_dinv_gold): D_inv, the
// fluxes of prim in the shared frame and, of a point the sweeps do not update,
// the published increment G(prim(U + dU)) - G(prim).  The fluxes are evaluated
// in R and go into gold[0..29]; D_inv is double.
template <typename R>
__device__ __forceinline__ void point_inputs(const DevCloud &d, int i, double *gold) {
    double p[5];
#pragma unroll
    for (int r = 0; r < 5; ++r) p[r] = d.prim[5 * (size_t)i + r];
    const bool swept = d.swept[i] != 0;
    const int cls = d.cls[i];
    if (swept && cls <= CLS_OUTER) {
        const double as = sqrt(1.40 * p[4] / p[0]);
        double gd[NDIR];
        if (cls <= CLS_WALL) {
#pragma unroll
            for (int dd = 0; dd < NDIR; ++dd) gd[dd] = dinv_term(d, i, dd, p[1 + (dd >> 1)], as);
            d.dinv[i] = dinv_combine(cls, d.delt[i], gd);
        } else {                                      // backup driver
#pragma unroll
            for (int dd = 0; dd < 5; ++dd) gd[dd] = dinv_term(d, i, dd, p[1 + (dd >> 1)], as, dd == 4 ? 5 : dd);
            d.dinv[i] = dinv_outer(d, i, gd);
        }
    }
    if (!d.shared_frame) return;
    FrameT<R> F0, F;
    load_frame(d.frame0, F0);
    R pr[5];
#pragma unroll
    for (int r = 0; r < 5; ++r) pr[r] = (R)p[r];
    FluxPreT<R> P;
    AxisTermsT<R> A[3];
    prim_terms(pr, F0, P, A);
#pragma unroll
    for (int dd = 0; dd < NDIR; ++dd) {
        R f[5];
        axis_flux(false, dd >> 1, (dd & 1) == 0, P, A[dd >> 1], R(0), R(0), f);
#pragma unroll
        for (int c = 0; c < 5; ++c) gold[5 * dd + c] = (double)f[c];
    }
    // increments at U + dU: of a point the sweeps leave alone, and (backup
    // driver) of every point before the sweeps
    for (int old = 0; old < 2; ++old) {
        if (old ? d.dg_old == nullptr : swept) continue;
        const double *du = (old ? d.dU_old : d.dUp) + 5 * (size_t)i;
        R U[5];
#pragma unroll
        for (int r = 0; r < 5; ++r) U[r] = (R)(du[r] + d.U[5 * (size_t)i + r]);
        load_frame(d.frame + 9 * (size_t)i, F);
        conserved_to_primitive(U, F, pr);
        prim_terms(pr, F0, P, A);
        const size_t o = DG_STRIDE * (size_t)i;
#pragma unroll
        for (int dd = 0; dd < NDIR; ++dd) {
            R f[5];
            axis_flux(false, dd >> 1, (dd & 1) == 0, P, A[dd >> 1], R(0), R(0), f);
#pragma unroll
            for (int c = 0; c < 5; ++c) {
                const double v = (double)(f[c] - (R)gold[5 * dd + c]);
                if (old) d.dg_old[o + DG_LIST * dd + c] = v;
                else d.dgf[o + DG_LIST * dd + c] = d.dgb[o + DG_LIST * dd + c] = v;
            }
        }
    }
}

// Least-squares moments of every point's conn (q_derivatives.f90:44-90), which
// do not change over a run: xx, yy, zz, xy, yz, zx, 1/det into d.qgeo when the
// handle is attached.  Weights come from d.wq (power != 0); with power = 0
// they are exactly 1, and delx*delx*1 rounds like the unweighted product.
// Also the points' coordinates into d.pos, where a neighbour's x, y, z and
// signal speed share one 32-byte sector.
__global__ void k_qgeo(DevCloud d, double *qgeo) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.n) return;
    const double xi = d.x[i], yi = d.y[i], zi = d.z[i];
    d.pos[4 * (size_t)i + 0] = xi;
    d.pos[4 * (size_t)i + 1] = yi;
    d.pos[4 * (size_t)i + 2] = zi;
    double xx = 0, yy = 0, zz = 0, xy = 0, yz = 0, zx = 0;
    const int nb = d.nbhs[i];
    for (int j = 0; j < nb; ++j) {
        const int k = d.conn[(size_t)MAX_CONN * i + j];
        const double w = d.wq ? d.wq[(size_t)MAX_CONN * i + j] : 1.0;
        const double delx = d.x[k] - xi, dely = d.y[k] - yi, delz = d.z[k] - zi;
        xx = xx + delx * delx * w;
        yy = yy + dely * dely * w;
        zz = zz + delz * delz * w;
        xy = xy + delx * dely * w;
        yz = yz + dely * delz * w;
        zx = zx + delz * delx * w;
    }
    const double det = xx * (yy * zz - yz * yz) - xy * (xy * zz - yz * zx) + zx * (xy * yz - yy * zx);
    double *g = qgeo + QGEO_STRIDE * (size_t)i;
    g[0] = xx;
    g[1] = yy;
    g[2] = zz;
    g[3] = xy;
    g[4] = yz;
    g[5] = zx;
    g[6] = 1.0 / det;
    g[7] = 0.0;
}

// eval_q_derivatives (q_derivatives.f90:25-110) and timestep_delt
// (timestep_delt.f90:227-259): five lanes per point, one per component of q,
// six points per warp.  What bounds it is the latency of the neighbours'
// gathers, so each lane has QD_BATCH neighbours' loads in flight.  The time
// step's neighbours are dealt out over the five lanes (a minimum does not
// depend on its order; a neighbour's signal speed was evaluated with its
// state, k_update).  600 points: 12 us against 32 with a thread per point and
// every neighbour's square roots; 62,400: 46 against 56; 1.1M: 0.60 against
// 0.67 ms.
constexpr int QD_THREADS = 128, QD_POINTS = QD_THREADS / 32 * 6, QD_BATCH = 5;
__global__ void __launch_bounds__(QD_THREADS) k_qderiv(const __grid_constant__ DevCloud d) {
    const int lane = threadIdx.x & 31, r = lane % 5;
    const int i0 = blockIdx.x * QD_POINTS + (threadIdx.x >> 5) * 6;
    const bool live = lane < 30 && i0 + lane / 5 < d.n;
    const int i = live ? i0 + lane / 5 : min(i0, d.n - 1);
    const double2 *pos = reinterpret_cast<const double2 *>(d.pos);   // (x, y), (z, speed)
    const double2 xyi = pos[2 * (size_t)i];
    const double xi = xyi.x, yi = xyi.y, zi = pos[2 * (size_t)i + 1].x;
    const double qi = d.q[5 * (size_t)i + r];
    double qmax = qi, qmin = qi, sx = 0.0, sy = 0.0, sz = 0.0, min_delt = 1.0;
    const int nb = d.nbhs[i];
    const int32_t *cn = d.conn + (size_t)MAX_CONN * i;
    for (int j0 = 0; j0 < nb; j0 += QD_BATCH) {
        int k[QD_BATCH];
        double2 xy[QD_BATCH], zs[QD_BATCH];
        double q[QD_BATCH];
#pragma unroll
        for (int b = 0; b < QD_BATCH; ++b) k[b] = j0 + b < nb ? cn[j0 + b] : i;
#pragma unroll
        for (int b = 0; b < QD_BATCH; ++b) {
            xy[b] = pos[2 * (size_t)k[b]];
            zs[b] = pos[2 * (size_t)k[b] + 1];
            q[b] = d.q[5 * (size_t)k[b] + r];
        }
        // the lane's own neighbour of the batch
        double2 xym = xy[0], zsm = zs[0];
#pragma unroll
        for (int b = 1; b < QD_BATCH; ++b) {
            xym = r == b ? xy[b] : xym;
            zsm = r == b ? zs[b] : zsm;
        }
#pragma unroll
        for (int b = 0; b < QD_BATCH; ++b) {
            if (j0 + b < nb) {
                const double w = d.wq ? d.wq[(size_t)MAX_CONN * i + j0 + b] : 1.0;
                const double delx = xy[b].x - xi, dely = xy[b].y - yi, delz = zs[b].x - zi;
                const double t = q[b] - qi;
                if (q[b] > qmax) qmax = q[b];
                if (q[b] < qmin) qmin = q[b];
                sx = sx + w * delx * t;
                sy = sy + w * dely * t;
                sz = sz + w * delz * t;
            }
        }
        if (j0 + r < nb) {
            const double delx = xym.x - xi, dely = xym.y - yi, delz = zsm.x - zi;
            const double dist = sqrt(delx * delx + dely * dely + delz * delz);
            const double delt = d.cfl * dist / zsm.y;       // timestep_delt.f90:235-253
            if (delt < min_delt) min_delt = delt;
        }
    }
    static_assert(QD_BATCH == 5, "a batch deals one neighbour to each lane of a point");
#pragma unroll
    for (int b = 1; b < 5; ++b) {
        const double o = __shfl_sync(FULL, min_delt, lane - r + (r + b) % 5);
        if (o < min_delt) min_delt = o;
    }
    if (!live) return;
    const double *g = d.qgeo + QGEO_STRIDE * (size_t)i;
    const double one_by_det = g[6];
#pragma unroll
    for (int a = 0; a < 3; ++a) d.dq[15 * (size_t)i + 3 * r + a] = cramer_num(a, g, sx, sy, sz) * one_by_det;
    d.qm[10 * (size_t)i + 2 * r + 0] = qmax;
    d.qm[10 * (size_t)i + 2 * r + 1] = qmin;
    if (r == 0) d.delt[i] = min_delt;
}

// eval_flux_residual (flux_residual.f90:40-81): one warp per point.  Lanes
// own the point's distinct neighbours: each reconstructs both ends of its
// pair once and evaluates the flux of every list the neighbour belongs to;
// then 30 lanes (list, component) sum the list terms in list order and solve
// the 3x3 least-squares system with the precomputed moments.
//
// R: the type of the reconstruction, limiter and flux arithmetic (float in
// mixed precision); the offsets, weights, list sums and 3x3 solves are double.
// One end j of a neighbour pair in straight-line code (reconstruct, flux_pre,
// axis_terms); ok is cleared where an argument is out of its range.
template <typename R>
__device__ __forceinline__ void end_core(const DevCloud &d, int j, R delx, R dely, R delz, const FrameT<R> &F, FluxPreT<R> &P,
                                         AxisTermsT<R> A[3], bool &ok) {
    const double *qj = d.q + 5 * (size_t)j, *dqj = d.dq + 15 * (size_t)j, *qmj = d.qm + 10 * (size_t)j;
    const R eps2 = (R)d.eps2[j];
    R qt[5], prim[5], yspb;
#pragma unroll
    for (int r = 0; r < 5; ++r) {
        const R q = (R)qj[r];
        const R temp = delx * (R)dqj[3 * r] + dely * (R)dqj[3 * r + 1] + delz * (R)dqj[3 * r + 2];
        qt[r] = q - R(0.5) * limiter_core(q, temp, (R)qmj[2 * r], (R)qmj[2 * r + 1], eps2, ok) * temp;
    }
    prim_core(qt, prim, ok);
    pre_core(prim, F, P, yspb, ok);
    axes_core(P, yspb, A, ok);
}
template <typename R>
__device__ __forceinline__ void end_general(const DevCloud &d, int j, R delx, R dely, R delz, const FrameT<R> &F,
                                            FluxPreT<R> &P, AxisTermsT<R> A[3]) {
    R prim[5];
    reconstruct<R>(d, j, delx, dely, delz, prim);
    flux_pre(prim, F, P);
#pragma unroll
    for (int a = 0; a < 3; ++a) axis_terms(P, a, A[a]);
}

// One end's fluxes for every list the slot is in, into T[(list * 32 + lane) * 5
// + component]: the first end's, then the second's less the first's.
template <typename R>
__device__ __forceinline__ void end_terms(int cls, int mask, int lane, const FluxPreT<R> &P, const AxisTermsT<R> A[3],
                                          bool second, double *T) {
    const bool wall = cls == CLS_WALL, octant = cls != CLS_INTERIOR;
    const R A3 = wall ? A[2].An : A[2].Ap, B3 = wall ? -A[2].B : A[2].B;
    for (; __any_sync(FULL, mask != 0); mask = mask_rest(mask)) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const int both = (mask >> (2 * a)) & 3;
            const bool pos = (both & 1) != 0;
            R f[5];
            axis_flux(octant && a < 2, a, pos, P, A[a], A3, B3, f);
            double *t = T + ((2 * a + (pos ? 0 : 1)) * MAX_SLOTS + lane) * 5;
            if (both) {
#pragma unroll
                for (int c = 0; c < 5; ++c) t[c] = second ? (double)(f[c] - (R)t[c]) : (double)f[c];
            }
        }
    }
}

// The terms with the operators, where an end's arguments left the range of the
// straight-line code.
template <typename R>
__device__ __noinline__ void end_terms_general(const DevCloud &d, int p, int j, R delx, R dely, R delz, int cls, int mask,
                                               int lane, bool second, double *T) {
    FrameT<R> F;
    load_frame(d.frame + 9 * (size_t)p, F);
    FluxPreT<R> P;
    AxisTermsT<R> A[3];
    end_general<R>(d, j, delx, dely, delz, F, P, A);
    end_terms<R>(cls, mask, lane, P, A, second, T);
}

// Bound by the FP64 pipe (58% busy) and the latency of the ends' gathers at 16
// warps per SM (prefetches into L1 for the neighbour's end or the next point
// gained nothing).  Blocks per SM the compiler must fit: four in FP64 (128
// registers; 1.1M points: three are 20% slower, five 6%), five in FP32 (62,400
// points: 0.26 ms against 0.28 with four and 0.26 with six).  The pair's ends go
// through one copy of the code: with both ends' code in a row the loop overran
// the instruction cache (1.1M points: 9.4 against 7.9 ms).  With the branch-free
// functions, storage order, the three axes side by side and the list's entries
// and moments read before the sums, 1.1M points take 5.0 ms against 10.7 ms
// before; 250k points in FP32 0.97 ms.
template <typename R>
constexpr int flux_blocks() { return sizeof(R) == 8 ? 4 : 5; }

//
// RS other than void (chain schedule): the first ceil(n / 128) blocks instead
// evaluate the sweep inputs, a thread per point (point_inputs<RS>), after
// marking their points' hand-off words DU_PENDING.
template <typename R, typename RS>
__global__ void __launch_bounds__(FLUX_WARPS * 32, flux_blocks<R>()) k_flux(const __grid_constant__ DevCloud d) {
    extern __shared__ double smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int first = 0;
    if constexpr (!std::is_void<RS>::value) {
        constexpr int PTS = FLUX_WARPS * 32;
        first = (d.n + PTS - 1) / PTS;
        if ((int)blockIdx.x < first) {
            const size_t i0 = (size_t)blockIdx.x * PTS, i1 = min(i0 + PTS, (size_t)d.n);
            const double pend = __longlong_as_double((long long)DU_PENDING);
            if (d.shared_frame)
                for (size_t w = DG_STRIDE * i0 + threadIdx.x; w < DG_STRIDE * i1; w += PTS) d.dgf[w] = d.dgb[w] = pend;
            for (size_t w = 5 * i0 + threadIdx.x; w < 5 * i1; w += PTS)
                if (d.swept[w / 5]) d.dUp[w] = d.dUn[w] = pend;
            __syncthreads();              // before the fixed increments over the marks
            // the fluxes' rows through shared memory, for whole-line stores
            // (an odd stride: no bank conflicts)
            constexpr int ROW = 31;
            static_assert(PTS * ROW <= FLUX_WARPS * FLUX_SMEM_PER_WARP, "rows fit the flux warps' memory");
            if (i0 + threadIdx.x < i1) point_inputs<RS>(d, (int)(i0 + threadIdx.x), smem + ROW * threadIdx.x);
            __syncthreads();
            if (d.shared_frame)
                for (int w = threadIdx.x; w < 30 * (int)(i1 - i0); w += PTS)
                    d.gold[30 * i0 + w] = smem[w / 30 * ROW + w % 30];
            return;
        }
    }
    double *T = smem + warp * FLUX_SMEM_PER_WARP;     // T[(dir*32 + slot)*5 + c]
    double *W = T + NDIR * MAX_SLOTS * 5;             // W[slot*3 + axis]
    const int dd = lane / 5, c = lane - 5 * (lane / 5);
    for (int p = (blockIdx.x - first) * FLUX_WARPS + warp; p < d.n; p += (gridDim.x - first) * FLUX_WARPS) {
        // read together: each would be a round trip of its own
        const int cls = d.cls[p], slots = d.nslot[p];
        const int slot_k = d.slot_nbr[(size_t)p * MAX_SLOTS + lane], slot_m = d.slot_mask[(size_t)p * MAX_SLOTS + lane];
        if (cls <= 2) {
            // lanes without a slot take the point itself and no list
            const bool have = lane < slots;
            const int k = have ? slot_k : p;
            const int mask = have ? slot_m : 0;
            Frame F;
            load_frame(d.frame + 9 * (size_t)p, F);
            const double delx = d.pos[4 * (size_t)k] - d.pos[4 * (size_t)p], dely = d.pos[4 * (size_t)k + 1] - d.pos[4 * (size_t)p + 1],
                         delz = d.pos[4 * (size_t)k + 2] - d.pos[4 * (size_t)p + 2];
            // dels*weights, delt*weights, deln*weights (weights 1 for power 0)
            const double w = d.wf ? d.wf[(size_t)MAX_SLOTS * p + lane] : 1.0;
            W[lane * 3 + 0] = (delx * F.t1[0] + dely * F.t1[1] + delz * F.t1[2]) * w;
            W[lane * 3 + 1] = (delx * F.t2[0] + dely * F.t2[1] + delz * F.t2[2]) * w;
            W[lane * 3 + 2] = (delx * F.n[0] + dely * F.n[1] + delz * F.n[2]) * w;
#pragma unroll 1
            for (int e = 0; e < 2; ++e) {
                const int j = e ? k : p;
                FluxPreT<R> P;
                AxisTermsT<R> A[3];
                FrameT<R> FR;
#pragma unroll
                for (int r = 0; r < 3; ++r) { FR.t1[r] = (R)F.t1[r]; FR.t2[r] = (R)F.t2[r]; FR.n[r] = (R)F.n[r]; }
                bool ok = true;
                end_core<R>(d, j, (R)delx, (R)dely, (R)delz, FR, P, A, ok);
                if (__all_sync(FULL, ok || !have)) end_terms<R>(cls, mask, lane, P, A, e != 0, T);
                else end_terms_general<R>(d, p, j, (R)delx, (R)dely, (R)delz, cls, mask, lane, e != 0, T);
            }
            // the lane's list (up to 27 entries of a byte, 28 apart), its first
            // entries and its moments, all before the sums that wait for them
            const int dl = lane < 30 ? dd : 0;
            const int cnt = lane < 30 ? d.list_cnt[(size_t)p * NDIR + dl] : 0;
            const uint32_t *ent = reinterpret_cast<const uint32_t *>(d.list_ent + ((size_t)p * NDIR + dl) * LIST_STRIDE);
            uint32_t e4[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) e4[q] = ent[q];
            const double *gp = d.geo + (size_t)p * GEO_STRIDE + dl * 8;
            double g[7];
#pragma unroll
            for (int r = 0; r < 7; ++r) g[r] = gp[r];
            __syncwarp();
            double G = 0.0;
            if (lane < 30) {
                double sx = 0.0, sy = 0.0, sz = 0.0;
                const double *t = T + dd * MAX_SLOTS * 5 + c;
                auto add = [&](uint32_t w, int j) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        if (j + q < cnt) {
                            const int s = (w >> (8 * q)) & 255;
                            const double v = t[s * 5];
                            sx = sx + v * W[s * 3 + 0];
                            sy = sy + v * W[s * 3 + 1];
                            sz = sz + v * W[s * 3 + 2];
                        }
                    }
                };
#pragma unroll
                for (int q = 0; q < 4; ++q) add(e4[q], 4 * q);
                for (int j = 16; j < cnt; j += 4) add(ent[j >> 2], j);
                const double num = cramer_select(dd >> 1, g, sx, sy, sz), det = g[G_DET];
                // outer_flux_dG*.f90:118-124 multiply by 1/det; the others divide
                const double y = rcp_rn(det);
                if (ieee_ok(fabs(det)) && ieee_num_ok(num)) G = (cls == CLS_OUTER) ? num * y : quot_rn(num, det, y);
                else G = (cls == CLS_OUTER) ? num * (1.0 / det) : num / det;
            }
            double gd[NDIR];
#pragma unroll
            for (int e = 0; e < NDIR; ++e) gd[e] = __shfl_sync(FULL, G, e * 5 + (lane % 5));
            if (lane < 5) {
                double r;
                if (cls == CLS_INTERIOR) r = gd[0] + gd[1] + gd[2] + gd[3] + gd[4] + gd[5];
                else if (cls == CLS_WALL) r = 2.0 * (gd[0] + gd[1] + gd[2] + gd[3] + gd[5]);
                else r = gd[0] + gd[1] + gd[2] + gd[3] + gd[4];
                d.flux_res[5 * (size_t)p + lane] = r;
            }
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------- D_inv and sweep inputs

// Fluxes of prim in the shared interior frame, all six directions.
__device__ __forceinline__ void flux6_frame0(const DevCloud &d, const double prim[5], double out[30]) {
    Frame F;
#pragma unroll
    for (int r = 0; r < 3; ++r) { F.t1[r] = d.frame0[r]; F.t2[r] = d.frame0[3 + r]; F.n[r] = d.frame0[6 + r]; }
    FluxPre P;
    flux_pre(prim, F, P);
    AxisTerms A[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) axis_terms(P, a, A[a]);
#pragma unroll
    for (int dd = 0; dd < NDIR; ++dd)
#pragma unroll
        for (int c = 0; c < 5; ++c) out[dd * 5 + c] = flux_component(dd, c, P, A);
}

// Before the sweeps (level and dataflow schedules): every published-increment
// word, and dU of every swept point, is set to DU_PENDING (coalesced
// grid-stride fill).
__global__ void k_pending(DevCloud d) {
    const double pend = __longlong_as_double((long long)DU_PENDING);
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    const size_t t0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t ng = (size_t)d.n * DG_STRIDE, nu = (size_t)d.n * 5;
    for (size_t w = t0; w < ng; w += stride) {
        d.dgf[w] = pend;
        d.dgb[w] = pend;
    }
    for (size_t w = t0; w < nu; w += stride) {
        if (d.swept[w / 5]) {
            d.dUp[w] = pend;
            d.dUn[w] = pend;
        }
    }
}

// implicit_D_inv_interior.f90:46-417 / implicit_D_inv_wall.f90:45-356 (see
// dinv_term); plus the sweep inputs that do not depend on the sweep: G(prim_k) in the shared frame for every point and the
// published increment G(prim(U_k + dU_k)) - G(prim_k) of points the sweeps
// never update (outer points, point 1), over the DU_PENDING that k_pending
// wrote there.
__global__ void __launch_bounds__(128) k_dinv_gold(DevCloud d) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.n) return;
    const int cls = d.cls[i];
    const double *p = d.prim + 5 * (size_t)i;
    if (d.swept[i] && cls <= CLS_WALL) {
        const double as = sqrt(1.40 * p[4] / p[0]);
        double gd[NDIR];
#pragma unroll
        for (int dd = 0; dd < NDIR; ++dd) gd[dd] = dinv_term(d, i, dd, p[1 + (dd >> 1)], as);
        d.dinv[i] = dinv_combine(cls, d.delt[i], gd);
    } else if (d.swept[i] && cls == CLS_OUTER) {   // backup driver
        const double as = sqrt(1.40 * p[4] / p[0]);
        double g5[5];
#pragma unroll
        for (int dd = 0; dd < 5; ++dd) g5[dd] = dinv_term(d, i, dd, p[1 + (dd >> 1)], as, dd == 4 ? 5 : dd);
        d.dinv[i] = dinv_outer(d, i, g5);
    }
    if (d.shared_frame) {
        double prim[5], gold[30];
#pragma unroll
        for (int r = 0; r < 5; ++r) prim[r] = p[r];
        flux6_frame0(d, prim, gold);
#pragma unroll
        for (int c = 0; c < 30; ++c) d.gold[30 * (size_t)i + c] = gold[c];
        if (!d.swept[i]) {
            double U[5], pn[5], gnew[30];
            Frame F;
            load_frame(d.frame + 9 * (size_t)i, F);
#pragma unroll
            for (int r = 0; r < 5; ++r) U[r] = d.dUp[5 * (size_t)i + r] + d.U[5 * (size_t)i + r];
            conserved_to_primitive(U, F, pn);
            flux6_frame0(d, pn, gnew);
#pragma unroll
            for (int c = 0; c < 30; ++c) {
                const double v = gnew[c] - gold[c];
                const size_t o = DG_STRIDE * (size_t)i + DG_LIST * (c / 5) + c % 5;
                d.dgf[o] = v;
                d.dgb[o] = v;
            }
        }
        if (d.dg_old) {   // backup driver: the increment from before the sweeps
            double U[5], pn[5], gnew[30];
            Frame F;
            load_frame(d.frame + 9 * (size_t)i, F);
#pragma unroll
            for (int r = 0; r < 5; ++r) U[r] = d.dU_old[5 * (size_t)i + r] + d.U[5 * (size_t)i + r];
            conserved_to_primitive(U, F, pn);
            flux6_frame0(d, pn, gnew);
#pragma unroll
            for (int c = 0; c < 30; ++c)
                d.dg_old[DG_STRIDE * (size_t)i + DG_LIST * (c / 5) + c % 5] = gnew[c] - gold[c];
        }
    }
}

// ---------------------------------------------------------------- LU-SGS sweeps

// Per-warp shared memory of the sweep kernels.  SweepStage holds everything a
// point reads that the sweep itself does not change (its terms, geometry,
// fluxes of prim in the shared frame, D_inv, U, frame, slot table); it is
// filled with cp.async, so the chain kernel loads the next point's stage
// while it works on the current one.
struct __align__(16) SweepStage {
    SweepEntry ent[SWEEP_MAX_ENTRIES];
    double geo[GEO_STRIDE];
    double gold[32];
    double U[6];
    double base[6];
    double frame[10];
    double dinv[2];
    int32_t slot_nbr[MAX_SLOTS];
    uint8_t slot_mask[MAX_SLOTS];
    uint32_t need;
    uint32_t old;                 // slots read from before the sweep (backup driver)
    int32_t pad[2];
};
constexpr int SW_T_DOUBLES = NDIR * MAX_SLOTS * 5;                  // term fluxes, >= SWEEP_MAX_ENTRIES * 5
constexpr int SWEEP_SMEM_BYTES = SW_T_DOUBLES * 8 + (int)sizeof(SweepStage);   // one stage
static_assert(SW_T_DOUBLES >= SWEEP_MAX_ENTRIES * 5, "T buffer too small");
static_assert(SW_T_DOUBLES * 8 >= SWEEP_MAX_ENTRIES * 5 * 8 + SWEEP_MAX_ENTRIES, "no room for the terms' flags");
static_assert(SW_T_DOUBLES == G0_DOUBLES && G0_DOUBLES % 2 == 0, "a g0 block is one T buffer of 16-byte pairs");
static_assert(SWEEP_MAX_ENTRIES <= 96, "entries are polled in three passes of 32");
static_assert(sizeof(SweepStage) % 16 == 0 && SWEEP_SMEM_BYTES % 16 == 0,
              "stage alignment");

enum SweepMode { MODE_LEVELS = 0, MODE_DATAFLOW = 1 };

__device__ __forceinline__ void cp_async16(void *s, const void *g) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(s)),
                 "l"(g)
                 : "memory");
}
__device__ __forceinline__ void cp_async8(void *s, const void *g) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(s)),
                 "l"(g)
                 : "memory");
}
__device__ __forceinline__ void cp_async4(void *s, const void *g) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(s)),
                 "l"(g)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_one() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

__device__ __forceinline__ int item_count(uint32_t cnt, int e) { return (int)((cnt >> (5 * e)) & 31u); }

// The record of point p for the level and dataflow schedules (the chain
// schedule reads precomputed ones).
__device__ __forceinline__ ChainItem make_item(const DevCloud &d, int p, bool forward) {
    ChainItem it;
    it.p = p;
    it.off = forward ? d.fwd_off[p] : d.bwd_off[p];
    const uint8_t *cnt = (forward ? d.fwd_cnt : d.bwd_cnt) + (size_t)p * NDIR;
    it.cnt = 0;
#pragma unroll
    for (int e = 0; e < NDIR; ++e) it.cnt |= (uint32_t)cnt[e] << (5 * e);
    it.info = (d.cls[p] == CLS_WALL ? CI_WALL : 0u) | (d.consumer_shared[p] ? CI_SHARED : 0u) | CI_PUBLISH |
              (d.cls[p] == CLS_SUPERSONIC ? CI_COPY : 0u) | (d.cls[p] == CLS_OUTER ? CI_OUTER : 0u);
    return it;
}

// Issue the cp.async copies of one point's stage (all lanes; caller commits).
// Every source is 16-byte aligned for the 16-byte copies: entries are 32-byte
// records, geo rows 384 bytes, gold rows 240 bytes, slot rows 128 / 32 bytes.
__device__ __forceinline__ void stage_issue(const DevCloud &d, const ChainItem &it, bool forward, int lane,
                                            SweepStage *st) {
    const size_t p = (size_t)it.p;
    int total = 0;
#pragma unroll
    for (int e = 0; e < NDIR; ++e) total += item_count(it.cnt, e);
    const char *es = reinterpret_cast<const char *>((forward ? d.fwd_ent : d.bwd_ent) + it.off);
    char *ed = reinterpret_cast<char *>(st->ent);
    for (int j = lane; j < 2 * total; j += 32) cp_async16(ed + 16 * j, es + 16 * j);
    if (lane < GEO_STRIDE / 2) cp_async16(st->geo + 2 * lane, d.geo + p * GEO_STRIDE + 2 * lane);
    if (lane < 15) cp_async16(st->gold + 2 * lane, d.gold + 30 * p + 2 * lane);
    if (lane < 5) {
        cp_async8(st->U + lane, d.U + 5 * p + lane);
        cp_async8(st->base + lane, (forward ? d.flux_res : d.dUp) + 5 * p + lane);
    } else if (lane < 14) {
        cp_async8(st->frame + (lane - 5), d.frame + 9 * p + (lane - 5));
    } else if (lane == 14) {
        cp_async8(st->dinv, d.dinv + p);
    } else if (!(it.info & CI_SHARED)) {
        if (lane < 23) cp_async16(st->slot_nbr + 4 * (lane - 15), d.slot_nbr + p * MAX_SLOTS + 4 * (lane - 15));
        else if (lane < 25) cp_async16(st->slot_mask + 16 * (lane - 23), d.sweep_slot_mask + p * MAX_SLOTS + 16 * (lane - 23));
        else if (lane == 25) cp_async4(&st->need, (forward ? d.fwd_need : d.bwd_need) + p);
        else if (lane == 26) cp_async4(&st->old, (forward ? d.fwd_old : d.bwd_old) + p);
    }
}

// Phase A of a point outside the shared frame, one lane per neighbour slot:
// the fluxes of the neighbour's state at the start of the sweep in the
// point's frame, for every list the slot is in, into
// T[(list * MAX_SLOTS + slot) * 5 + component].  The sweep runs it in place,
// or k_g0 runs it for all such points before the sweeps (the same code, so
// the same bits).
template <typename R>
__device__ __forceinline__ void neighbour_fluxes(const DevCloud &d, int cls, const FrameT<R> &Fp, int k_slot,
                                                 int mask_slot, int lane, double *T) {
    R po[5];
#pragma unroll
    for (int r = 0; r < 5; ++r) po[r] = (R)d.prim[5 * (size_t)k_slot + r];
    FluxPreT<R> Po;
    flux_pre(po, Fp, Po);
    int axes = 0;
#pragma unroll
    for (int e = 0; e < NDIR; ++e)
        if (mask_slot & (1 << e)) axes |= kind_axes(flux_kind(cls, e));
    AxisTermsT<R> Ao[3];
#pragma unroll
    for (int a = 0; a < 3; ++a)
        if (axes & (1 << a)) axis_terms(Po, a, Ao[a]);
    for (int e = 0; e < NDIR; ++e) {
        if (!(mask_slot & (1 << e))) continue;
        const int kind = flux_kind(cls, e);
#pragma unroll
        for (int cc = 0; cc < 5; ++cc)
            T[(e * MAX_SLOTS + lane) * 5 + cc] = (double)flux_component(kind, cc, Po, Ao);
    }
}

// Phase A of every g0 point (Topology::g0_pts) from the state at the start
// of the iteration, which both sweeps read: one warp per point.
template <typename R>
__global__ void __launch_bounds__(128) k_g0(DevCloud d) {
    const int w = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (w >= d.n_g0) return;
    const int p = d.g0_pts[w];
    if (lane >= d.nslot[p]) return;
    const int mask = d.sweep_slot_mask[(size_t)p * MAX_SLOTS + lane];
    if (!mask) return;
    FrameT<R> Fp;
    load_frame(d.frame + 9 * (size_t)p, Fp);
    neighbour_fluxes<R>(d, d.cls[p], Fp, d.slot_nbr[(size_t)p * MAX_SLOTS + lane], mask, lane,
                        d.g0 + (size_t)w * G0_DOUBLES);
}

// One point of the forward (LdelU) or backward (UdelU) sweep, processed by
// one warp (implicit_forward_and_reverse_sweeps.f90:30-37 / :61-68), from its
// stage in shared memory.
//
// Phase A (no dependency on the sweep): points outside the shared frame
// evaluate G(prim_k) of their neighbours.  Phase B: collect the neighbours'
// increments as they are published (points in the shared frame: the
// published flux increments; others: dU_k, then G(prim(U_k + dU_k)) -
// G(prim_k)).  Phase C: sum each list in list order (30 lanes: list x
// component), solve the 3x3 systems, update dU and publish this point's own
// flux increment.
template <int MODE, typename R>
__device__ void sweep_point(const DevCloud &d, const ChainItem &it, const SweepStage *st, bool forward, int lane,
                            double *T) {
    const int p = it.p;
    const bool wall = (it.info & CI_WALL) != 0;
    const bool shared = (it.info & CI_SHARED) != 0;
    const bool copy = (it.info & CI_COPY) != 0;       // supersonic point
    const bool outer = (it.info & CI_OUTER) != 0;     // backup driver
    const bool hold = p + 1 == d.withhold1;           // failure-detection hook: publish nothing
    const int cls = wall ? CLS_WALL : (outer ? CLS_OUTER : CLS_INTERIOR);
    const SweepEntry *E = st->ent;
    const int dd = lane / 5, c = lane - 5 * (lane / 5);
    int total = 0, lo = 0, hi = 0;
#pragma unroll
    for (int e = 0; e < NDIR; ++e) {
        const int ce = item_count(it.cnt, e);
        if (e < dd) lo += ce;
        if (e <= dd) hi += ce;
        total += ce;
    }

    // ---- phase A
    double g[7] = {0, 0, 0, 0, 0, 0, 1.0};
    double gold = 0.0;
    if (lane < 30) {
        const int grow = (outer && dd == 4) ? 5 : dd;   // outer z+ over conn: row 5
#pragma unroll
        for (int r = 0; r < 7; ++r) g[r] = st->geo[grow * 8 + r];
        gold = st->gold[lane];
    }
    double dinv = 0.0, base5 = 0.0;
    if (lane < 5) {
        dinv = st->dinv[0];
        base5 = st->base[lane];
    }
    // inputs the concurrent flux kernel had not produced when the stage was copied
    if (lane < 30 && is_pending(gold)) gold = poll_word(d.gold + 30 * (size_t)p + lane, d);
    if (lane < 5 && !copy) {
        if (is_pending(dinv)) dinv = poll_word(d.dinv + p, d);
        if (is_pending(base5)) base5 = poll_word((forward ? d.flux_res : d.dUp) + 5 * (size_t)p + lane, d);
    }
    double Up[5];
#pragma unroll
    for (int r = 0; r < 5; ++r) Up[r] = st->U[r];
    FrameT<R> Fp;
    load_frame(st->frame, Fp);
    double dnew = 0.0;
    if (copy) {
        // implicit_forward_and_reverse_sweeps.f90:38-51 / :69-82: the
        // nearest neighbour's increment, updated earlier in this sweep or
        // from before it
        if (lane < 5) {
            const int q = E[0].k;
            double *dst = (forward ? d.dUp : d.dUn) + 5 * (size_t)p + lane;
            if (q >= 0)
                dnew = (E[0].pad & ENT_COPY_NEW) ? poll_word((forward ? d.dUp : d.dUn) + 5 * (size_t)q + lane, d)
                                                 : d.dU_old[5 * (size_t)q + lane];
            if (!hold) st_relaxed_f64(dst, dnew);
        }
    } else {
        double sx = 0.0, sy = 0.0, sz = 0.0;   // phase C's list sums
        const uint32_t need = shared ? 0u : st->need;
        const bool mine = !shared && (need >> lane) & 1u;
        int k_slot = 0, mask_slot = 0;
        if (mine) {
            k_slot = st->slot_nbr[lane];
            mask_slot = st->slot_mask[lane];
            neighbour_fluxes<R>(d, cls, Fp, k_slot, mask_slot, lane, T);
        }

        // ---- phase B
        // The list sums of phase C run in list order from `pos`; in the shared
        // frame they advance over the terms that have landed while later
        // ones are still awaited, so only the terms after the last arrival
        // remain once it lands (the additions keep their order).
        int pos = lo;
        if (shared) {
            // lane owns entries lane, lane+32, lane+64; all their loads are in
            // flight together, re-polling only the ones still pending; a
            // landed term's flag (past the 96 terms' values in T) tells the
            // summing lanes it is there
            const double *src = forward ? d.dgf : d.dgb;
            uint8_t *rdy = reinterpret_cast<uint8_t *>(T + 5 * SWEEP_MAX_ENTRIES);
            uint32_t pend = 0;
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const int j = lane + 32 * q;
                if (j >= total) continue;
                pend |= 1u << q;
                rdy[j] = 0;
            }
            int spins = 0;
            for (;;) {
                if (pend) {
                    unsigned long long v[3][5];
#pragma unroll
                    for (int q = 0; q < 3; ++q) {
                        if (!((pend >> q) & 1u)) continue;
                        const int j = lane + 32 * q;
                        // backup driver: a term from before the sweep reads dg_old
                        const double *base = (E[j].pad & ENT_OLD) ? d.dg_old : src;
                        const double *gs = base + DG_STRIDE * (size_t)E[j].k + DG_LIST * (E[j].pad & 255);
                        ld_relaxed_v2(gs, v[q][0], v[q][1]);
                        ld_relaxed_v2(gs + 2, v[q][2], v[q][3]);
                        v[q][4] = ld_relaxed_b64(gs + 4);
                    }
#pragma unroll
                    for (int q = 0; q < 3; ++q) {
                        if (!((pend >> q) & 1u) || !ready5(v[q])) continue;
                        const int j = lane + 32 * q;
#pragma unroll
                        for (int cc = 0; cc < 5; ++cc) T[j * 5 + cc] = __longlong_as_double(v[q][cc]);
                        rdy[j] = 1;
                        pend &= ~(1u << q);
                    }
                    if (pend && !spin_continue(spins, d)) {
                        // the wait ran out (d.err is set): the terms stay unset
#pragma unroll
                        for (int q = 0; q < 3; ++q)
                            if ((pend >> q) & 1u) rdy[lane + 32 * q] = 1;
                        pend = 0;
                    }
                }
                __syncwarp();
                if (__all_sync(FULL, pend == 0)) break;
                if (lane < 30) {
                    while (pos < hi && rdy[pos]) {
                        const double t = T[pos * 5 + c];
                        sx = sx + t * E[pos].w[0];
                        sy = sy + t * E[pos].w[1];
                        sz = sz + t * E[pos].w[2];
                        ++pos;
                    }
                }
                __syncwarp();
            }
        } else {
            FluxPreT<R> Pn;
            AxisTermsT<R> An[3];
            if (mine) {
                const bool old = (st->old >> lane) & 1u;   // backup driver: from before the sweep
                const double *dsrc = (old ? d.dU_old : (forward ? d.dUp : d.dUn)) + 5 * (size_t)k_slot;
                unsigned long long v[5];
                int spins = 0;
                do {
#pragma unroll
                    for (int r = 0; r < 5; ++r) v[r] = ld_relaxed_b64(dsrc + r);
                } while (!ready5(v) && spin_continue(spins, d));
                R U[5], pn[5];
#pragma unroll
                for (int r = 0; r < 5; ++r) U[r] = (R)(__longlong_as_double(v[r]) + d.U[5 * (size_t)k_slot + r]);
                FrameT<R> Fk;
                load_frame(d.frame + 9 * (size_t)k_slot, Fk);
                conserved_to_primitive(U, Fk, pn);
                flux_pre(pn, Fp, Pn);
                int axes = 0;
#pragma unroll
                for (int e = 0; e < NDIR; ++e)
                    if (mask_slot & (1 << e)) axes |= kind_axes(flux_kind(cls, e));
#pragma unroll
                for (int a = 0; a < 3; ++a)
                    if (axes & (1 << a)) axis_terms(Pn, a, An[a]);
            }
            if (mine) {
                for (int e = 0; e < NDIR; ++e) {
                    if (!(mask_slot & (1 << e))) continue;
                    const int kind = flux_kind(cls, e);
#pragma unroll
                    for (int cc = 0; cc < 5; ++cc) {
                        double *t = &T[(e * MAX_SLOTS + lane) * 5 + cc];
                        *t = (double)(flux_component(kind, cc, Pn, An) - (R)*t);
                    }
                }
            }
        }
        __syncwarp();

        // ---- phase C (from pos: the terms not yet summed)
        double G = 0.0;
        if (lane < 30) {
            // unrolled so the next terms' shared-memory loads overlap; the
            // additions keep their order
#pragma unroll 4
            for (int jj = pos; jj < hi; ++jj) {
                const double t = shared ? T[jj * 5 + c] : T[(dd * MAX_SLOTS + ((E[jj].pad >> 8) & 255)) * 5 + c];
                sx = sx + t * E[jj].w[0];
                sy = sy + t * E[jj].w[1];
                sz = sz + t * E[jj].w[2];
            }
        }
        if (lane < 30) G = cramer_num(dd >> 1, g, sx, sy, sz) / g[6];
        double gd[NDIR];
#pragma unroll
        for (int e = 0; e < NDIR; ++e) gd[e] = __shfl_sync(FULL, G, e * 5 + (lane % 5));
        if (lane < 5) {
            double lu;
            if (wall) lu = 2.0 * (gd[0] + gd[1] + gd[2] + gd[3] + gd[5]);
            else if (outer) lu = gd[0] + gd[1] + gd[2] + gd[3] + gd[4];   // *_sweep_outer.f90:406
            else lu = gd[0] + gd[1] + gd[2] + gd[3] + gd[4] + gd[5];
            if (forward) {
                dnew = -(dinv * (base5 + lu));
                if (!hold) st_relaxed_f64(d.dUp + 5 * (size_t)p + lane, dnew);
            } else {
                dnew = base5 - dinv * lu;
                if (!hold) st_relaxed_f64(d.dUn + 5 * (size_t)p + lane, dnew);
            }
        }
    }
    if (d.shared_frame) {
        // publish this point's increment for the consumers in the shared frame
        R U[5], pn[5];
#pragma unroll
        for (int r = 0; r < 5; ++r) U[r] = (R)(__shfl_sync(FULL, dnew, r) + Up[r]);
        if (lane < 30) {
            conserved_to_primitive(U, Fp, pn);
            FrameT<R> F0;
            load_frame(d.frame0, F0);
            FluxPreT<R> P;
            flux_pre(pn, F0, P);
            AxisTermsT<R> At;
            axis_terms(P, dd >> 1, At);
            const double v = (double)(flux_component(dd, c, P, At, At, At) - (R)gold);
            if ((it.info & CI_PUBLISH) && !hold)
                st_relaxed_f64((forward ? d.dgf : d.dgb) + DG_STRIDE * (size_t)p + DG_LIST * dd + c, v);
        }
    }
    __syncwarp();
}

// Stage one point synchronously and sweep it (level and dataflow schedules).
template <int MODE>
__device__ __forceinline__ void sweep_point_sync(const DevCloud &d, int p, bool forward, int lane, char *smb) {
    double *T = reinterpret_cast<double *>(smb);
    SweepStage *st = reinterpret_cast<SweepStage *>(smb + SW_T_DOUBLES * 8);
    const ChainItem it = make_item(d, p, forward);
    stage_issue(d, it, forward, lane, st);
    cp_async_commit();
    cp_async_wait_all();
    __syncwarp();
    sweep_point<MODE, double>(d, it, st, forward, lane, T);
}

// Level-synchronous sweep in one CTA: the points of a level are independent
// (none reads another's increment), so warps take them in parallel and a
// block barrier separates levels; every poll succeeds at once.
__global__ void __launch_bounds__(SWEEP_THREADS, 1) k_sweep_levels(DevCloud d, int forward) {
    extern __shared__ double smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    char *smb = reinterpret_cast<char *>(smem) + warp * SWEEP_SMEM_BYTES;
    const int nl = forward ? d.n_fwd_levels : d.n_bwd_levels;
    const int32_t *lptr = forward ? d.fwd_lvl_ptr : d.bwd_lvl_ptr;
    const int32_t *lpts = forward ? d.fwd_lvl_pts : d.bwd_lvl_pts;
    for (int l = 0; l < nl; ++l) {
        const int a = lptr[l], b = lptr[l + 1];
        for (int idx = a + warp; idx < b; idx += SWEEP_WARPS)
            sweep_point_sync<MODE_LEVELS>(d, lpts[idx], forward != 0, lane, smb);
        __syncthreads();
    }
}

// Dataflow sweep over many SMs: each warp takes the next point of the
// level-major (topological) order from a global counter and polls for the
// increments it reads.  A point's dependencies are always taken before it by
// warps that are already running, so the polls end; each is bounded anyway.
constexpr int DF_WARPS = 4;

__global__ void __launch_bounds__(DF_WARPS * 32) k_sweep_df(DevCloud d, int forward) {
    extern __shared__ double smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    char *smb = reinterpret_cast<char *>(smem) + warp * SWEEP_SMEM_BYTES;
    int *counter = d.sweep_counter + (forward ? 0 : 1);
    const int32_t *order = forward ? d.fwd_lvl_pts : d.bwd_lvl_pts;
    const int total = d.n_swept;
    for (;;) {
        int idx = 0;
        if (lane == 0) idx = atomicAdd(counter, 1);
        idx = __shfl_sync(FULL, idx, 0);
        if (idx >= total) break;
        sweep_point_sync<MODE_DATAFLOW>(d, order[idx], forward != 0, lane, smb);
    }
}

}  // namespace mfcfd

#include "mfcfd_chain.cuh"

namespace mfcfd {

// Residency.  Every wait of a sweep is for a point of the same sweep, so all
// blocks of the chain sweeps running at once have to fit the device together.
// They are counted in slots of a sixth of an SM: a 4-warp block takes 2 in
// mixed precision (three per SM: at most 168 registers and 76 KB of shared
// memory), 3 in FP64 (two per SM: 254 registers, no spills), or 2 in the dense
// FP64 build (168 registers, 100 bytes spilled), which a cloud takes whose teams
// need more than two blocks per SM (1.1M points, 396 teams of four: 27.9 ms
// per iteration against 31.6 as teams of two without the spills).  The sweeps at
// once take at most 6 * (SMs - CH_FREE_SMS) slots, a block half an SM at least
// where they differ in size (SlotPool); the other SMs' room is for the
// kernels of other handles between their sweeps.
constexpr int CH_FREE_SMS = 16;

template <typename R, bool FOLD, bool DENSE, bool AXES>
__global__ void __launch_bounds__(CH_WPB * 32, DENSE ? 3 : 2) k_sweep_chain(const __grid_constant__ DevCloud d, int forward) {
    chain_sweep<R, FOLD, AXES>(d, forward, blockIdx.x);
}

// The chain sweeps of a group of clouds in one launch: blocks
// [block_start[c], block_start[c + 1]) are cloud c's.  The clouds share
// nothing; a block finds its cloud and runs that cloud's schedule as the
// single-cloud kernel would.  The group lives in the launch's parameters, so
// every block reads its cloud's pointers from the constant bank.
template <typename R, bool FOLD, bool DENSE, bool AXES>
__global__ void __launch_bounds__(CH_WPB * 32, DENSE ? 3 : 2)
    k_sweep_chain_group(const __grid_constant__ ChainGroup g, int forward) {
    int c = 0;
    while (c + 1 < g.count && (int)blockIdx.x >= g.block_start[c + 1]) ++c;
    chain_sweep<R, FOLD, AXES>(g.cloud[c], forward, (int)blockIdx.x - g.block_start[c]);
}

// three blocks per SM: 228 KB of shared memory, 1 KB of it reserved per block
static_assert(3 * (chain_smem_bytes(1) + 1024) <= 228 * 1024 && 3 * (chain_smem_bytes(2) + 1024) <= 228 * 1024 &&
                  3 * (chain_smem_bytes(4) + 1024) <= 228 * 1024,
              "three chain blocks per SM");
// A spread chain block asks for this much shared memory, so that no second
// block fits beside it (2 x (116 + 1) KB > 228 KB) and each of its four
// warps has one of the SM's four sub-partitions to itself.
constexpr int CHAIN_SPREAD_SMEM = 116 * 1024;
static_assert(2 * (CHAIN_SPREAD_SMEM + 1024) > 228 * 1024 && CHAIN_SPREAD_SMEM >= chain_smem_bytes(2),
              "a spread block holds its SM alone");

static int chain_smem(const ChainShape &c) { return c.spread ? CHAIN_SPREAD_SMEM : chain_smem_bytes(c.team); }

// ---------------------------------------------------------------- state update

// state_update_implicit.f90:119-152 + 189-191 (or state_update.f90:29-78
// under MFCFD_UPDATE_EXPLICIT), then the next iteration's
// compute_conserved_vector / eval_q_variables into the other U/q buffer.
__global__ void k_update(DevCloud d, double *U_next, double *q_next) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.n) return;
    const int cls = d.cls[i];
    Frame F;
    load_frame(d.frame + 9 * (size_t)i, F);
    double U[5], dn[5], p[5];
#pragma unroll
    for (int r = 0; r < 5; ++r) dn[r] = d.dUn[5 * (size_t)i + r];
    double res = 0.0;
    const bool expl = d.update_variant == MFCFD_UPDATE_EXPLICIT;
    if (cls == CLS_WALL || cls == CLS_INTERIOR) {
        const double temp = d.U[5 * (size_t)i];
#pragma unroll
        for (int r = 0; r < 5; ++r) U[r] = d.U[5 * (size_t)i + r] + dn[r];
        if (expl && cls == CLS_WALL) U[3] = 0.0;   // state_update.f90:37
        res = (U[0] - temp) * (U[0] - temp);
        conserved_to_primitive(U, F, p);
    } else if (cls == CLS_OUTER) {
        double pc[5];
#pragma unroll
        for (int r = 0; r < 5; ++r) pc[r] = d.prim[5 * (size_t)i + r];
        conserved_vector_Ubar(pc, F, d.rho_inf, d.u1_inf, d.u2_inf, d.u3_inf, d.pr_inf, U);
        if (expl) {   // state_update.f90:55-58
            const double dt = d.delt[i];
#pragma unroll
            for (int r = 0; r < 5; ++r) U[r] = U[r] - dt * d.flux_res[5 * (size_t)i + r];
        } else {
#pragma unroll
            for (int r = 0; r < 5; ++r) U[r] = U[r] + dn[r];
        }
        conserved_to_primitive(U, F, p);
    } else {
#pragma unroll
        for (int r = 0; r < 5; ++r) p[r] = d.prim[5 * (size_t)i + r];
    }
    d.res_sqr[i] = res;
    d.pos[4 * (size_t)i + 3] = signal_speed(p);
    double Un[5], qn[5];
    primitive_to_rotated_conserved(p, F, Un);
    primitive_to_q(p, qn);
#pragma unroll
    for (int r = 0; r < 5; ++r) {
        d.prim[5 * (size_t)i + r] = p[r];
        d.dUp[5 * (size_t)i + r] = dn[r];
        U_next[5 * (size_t)i + r] = Un[r];
        q_next[5 * (size_t)i + r] = qn[r];
    }
}

// Supersonic points after the state update (state_update_implicit.f90:
// 63-94): outlets, then inlets, each in index order, take the new state of
// their nearest non-wall neighbour.  One thread, in that order, since a
// source may be a supersonic point copied just before; then their next U
// and q.
__global__ void k_update_ss(DevCloud d, double *U_next, double *q_next) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    for (int j = 0; j < d.n_ss; ++j) {
        const int k = d.ss_pts[j], src = d.ss_src[j];
        double p[5];
#pragma unroll
        for (int r = 0; r < 5; ++r) {
            p[r] = src >= 0 ? d.prim[5 * (size_t)src + r] : 0.0;
            d.prim[5 * (size_t)k + r] = p[r];
        }
        d.pos[4 * (size_t)k + 3] = signal_speed(p);
        Frame F;
        load_frame(d.frame + 9 * (size_t)k, F);
        double Un[5], qn[5];
        primitive_to_rotated_conserved(p, F, Un);
        primitive_to_q(p, qn);
#pragma unroll
        for (int r = 0; r < 5; ++r) {
            U_next[5 * (size_t)k + r] = Un[r];
            q_next[5 * (size_t)k + r] = qn[r];
        }
    }
}

// res_new = sqrt(sum over wall, interior of (dU1)^2) / N
// (state_update_implicit.f90:124-129, 187).  Fixed two-pass tree order, so
// the value is deterministic; it differs from the reference's left-to-right
// sum only by summation rounding.
__global__ void k_reduce_partial(DevCloud d) {
    __shared__ double s[RED_THREADS];
    const int per = (d.n_res + gridDim.x - 1) / gridDim.x;
    const int a = blockIdx.x * per, b = min(d.n_res, a + per);
    double acc = 0.0;
    for (int j = a + threadIdx.x; j < b; j += RED_THREADS) acc += d.res_sqr[d.res_order[j]];
    s[threadIdx.x] = acc;
    __syncthreads();
    for (int w = RED_THREADS / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) s[threadIdx.x] += s[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) d.partial[blockIdx.x] = s[0];
}

__global__ void k_reduce_final(DevCloud d, int nblocks, int slot) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    double acc = 0.0;
    for (int b = 0; b < nblocks; ++b) acc += d.partial[b];
    d.res_dev[slot] = sqrt(acc) / (double)d.n;
}

// ---------------------------------------------------------------- forces

// F = -sum over wall points of (p_i - p_inf) A_i nor_i, one block: thread t
// sums the wall points t, t + 256, ... in index order, then a fixed tree;
// A_i from area (per point) or area_each.  out[0..2] = F.
__global__ void __launch_bounds__(RED_THREADS) k_forces(DevCloud d, double area_each, const double *area,
                                                          double *out) {
    __shared__ double s[3][RED_THREADS];
    double f[3] = {0.0, 0.0, 0.0};
    for (int j = threadIdx.x; j < d.n_wall; j += RED_THREADS) {
        const int i = d.res_order[j];          // wall points first, index order
        const double a = area ? area[i] : area_each;
        const double dp = d.prim[5 * (size_t)i + 4] - d.pr_inf;
#pragma unroll
        for (int r = 0; r < 3; ++r) f[r] = f[r] - dp * a * d.frame[9 * (size_t)i + 6 + r];
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) s[r][threadIdx.x] = f[r];
    __syncthreads();
    for (int w = RED_THREADS / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w)
#pragma unroll
            for (int r = 0; r < 3; ++r) s[r][threadIdx.x] += s[r][threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x < 3) out[threadIdx.x] = s[threadIdx.x][0];
}

cudaError_t launch_forces(const DevCloud &d, cudaStream_t s, double area_each, const double *area, double *out) {
    k_forces<<<1, RED_THREADS, 0, s>>>(d, area_each, area, out);
    return cudaGetLastError();
}

// ---------------------------------------------------------------- launchers

int device_sms(int device) {
    static std::mutex mu;
    static int cache[256] = {0};
    if (device < 0 || device >= 256) return 1;
    std::lock_guard<std::mutex> lock(mu);
    if (!cache[device]) {
        int sms = 0;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || sms < 1) {
            (void)cudaGetLastError();
            sms = 1;
        }
        cache[device] = sms;
    }
    return cache[device];
}

// Mixed precision (MIXED, MIXED_DC): each sweep term's weight with its list's
// 3x3 least-squares solve folded in.  The list's derivative is num(axis,
// moments, sum w_j t_j) / det, linear in the sums, so every term gets one
// weight (cofactors . w_j) / det, in FP64, and the sweep sums w_j t_j
// directly.  fold: the three weights are saved first when `saved` is given
// (3 per term), then replaced; !fold: put back from `saved`.
__global__ void k_fold_terms(DevCloud d, int dir, double *saved, int fold) {
    const int *off = dir == 0 ? d.fwd_off : d.bwd_off;
    SweepEntry *ent = const_cast<SweepEntry *>(dir == 0 ? d.fwd_ent : d.bwd_ent);
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < d.n; p += gridDim.x * blockDim.x) {
        for (int e = off[p]; e < off[p + 1]; ++e) {
            SweepEntry &E = ent[e];
            if (E.pad & ENT_COPY) continue;
            if (!fold) {
                E.w[0] = saved[3 * (size_t)e];
                E.w[1] = saved[3 * (size_t)e + 1];
                E.w[2] = saved[3 * (size_t)e + 2];
                continue;
            }
            if (saved) {
                saved[3 * (size_t)e] = E.w[0];
                saved[3 * (size_t)e + 1] = E.w[1];
                saved[3 * (size_t)e + 2] = E.w[2];
            }
            const int dd = E.pad & 255;
            const bool outer_zp = d.sweep_variant == MFCFD_SWEEPS_BACKUP && d.cls[p] == CLS_OUTER && dd == 4;
            const double *g = d.geo + (size_t)p * GEO_STRIDE + (outer_zp ? 5 : dd) * 8;
            const double xx = g[G_XX], yy = g[G_YY], zz = g[G_ZZ], xy = g[G_XY], yz = g[G_YZ], zx = g[G_ZX];
            double a, b, c;
            if (dd / 2 == 0) { a = yy * zz - yz * yz; b = -(xy * zz - zx * yz); c = xy * yz - zx * yy; }
            else if (dd / 2 == 1) { a = -(xy * zz - zx * yz); b = xx * zz - zx * zx; c = -(xx * yz - xy * zx); }
            else { a = xy * yz - zx * yy; b = -(xx * yz - zx * xy); c = xx * yy - xy * xy; }
            const double w = (a * E.w[0] + b * E.w[1] + c * E.w[2]) / g[G_DET];
            E.w[0] = w;
            E.w[1] = 0.0;
            E.w[2] = 0.0;
        }
    }
}

cudaError_t launch_fold_terms(const DevCloud &d, double *const saved[2], bool fold, cudaStream_t s) {
    const int grid = (d.n + 255) / 256;
    for (int dir = 0; dir < 2; ++dir) k_fold_terms<<<grid, 256, 0, s>>>(d, dir, saved[dir], fold ? 1 : 0);
    return cudaGetLastError();
}

int reduction_blocks(int n) {
    int b = (n + 4095) / 4096;
    return b < 1 ? 1 : (b > 1024 ? 1024 : b);
}

// ---------------------------------------------------------------- allocation-free residual

// Scratch of mfcfd_residual_noalloc: one partial sum per reduction block plus
// the result slot.  A file-scope device array, so that entry point never
// allocates; 8 KB that every GPU loading the library holds until exit.
constexpr int NOALLOC_BLOCKS = MFCFD_NOALLOC_MAX_TERMS / 4096;
static __device__ __align__(256) double g_noalloc_scratch[NOALLOC_BLOCKS + 1];

// Device address of g_noalloc_scratch, looked up once per device.  In host
// code the symbol names a host-side stand-in, not device memory, so kernels
// must be given this address instead.
static std::mutex g_noalloc_mu;
static double *g_noalloc_ptr[256] = {nullptr};

int residual_noalloc(const DevCloud &d, cudaStream_t s, double *res_new, std::string &err) {
    if (d.n_res > MFCFD_NOALLOC_MAX_TERMS) {
        err = "mfcfd_residual_noalloc handles at most " + std::to_string(MFCFD_NOALLOC_MAX_TERMS) +
              " residual terms; this cloud has " + std::to_string(d.n_res);
        return MFCFD_ERR_UNSUPPORTED;
    }
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= 256) {
        err = std::string("cudaGetDevice: ") + cudaGetErrorString(e);
        return MFCFD_ERR_CUDA;
    }
    double *scratch = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_noalloc_mu);
        if (!g_noalloc_ptr[dev]) {
            void *p = nullptr;
            e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
            if (e != cudaSuccess) {
                err = std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e);
                return MFCFD_ERR_CUDA;
            }
            g_noalloc_ptr[dev] = static_cast<double *>(p);
        }
        scratch = g_noalloc_ptr[dev];
    }
    // Same partition as the iteration's own reduction (4096 terms a block),
    // so the value is the one mfcfd_fpi_step returned.  Every partial that
    // k_reduce_final reads is written first, so nothing needs clearing.
    int blocks = (d.n_res + 4095) / 4096;
    if (blocks < 1) blocks = 1;
    DevCloud dc = d;
    dc.partial = scratch;
    dc.res_dev = scratch + NOALLOC_BLOCKS;
    k_reduce_partial<<<blocks, RED_THREADS, 0, s>>>(dc);
    k_reduce_final<<<1, 32, 0, s>>>(dc, blocks, 0);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(res_new, scratch + NOALLOC_BLOCKS, sizeof(double),
                                              cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        err = std::string("residual_noalloc: ") + cudaGetErrorString(e);
        return MFCFD_ERR_CUDA;
    }
    return MFCFD_OK;
}

// f(kernel, its group form, whether three blocks share an SM) for each form of
// the chain sweep.
template <typename F>
static void each_chain_kernel(F f) {
    f(k_sweep_chain<double, false, false, true>, k_sweep_chain_group<double, false, false, true>, false);
    f(k_sweep_chain<double, false, true, true>, k_sweep_chain_group<double, false, true, true>, true);
    f(k_sweep_chain<float, true, true, true>, k_sweep_chain_group<float, true, true, true>, true);
    f(k_sweep_chain<double, false, false, false>, k_sweep_chain_group<double, false, false, false>, false);
    f(k_sweep_chain<double, false, true, false>, k_sweep_chain_group<double, false, true, false>, true);
    f(k_sweep_chain<float, true, true, false>, k_sweep_chain_group<float, true, true, false>, true);
}

// Sets the kernels' shared-memory limits once per device.
static void set_attributes(int device) {
    static std::mutex mu;
    static bool done[256] = {false};
    std::lock_guard<std::mutex> lock(mu);
    if (device < 0 || device >= 256 || done[device]) return;
    auto flux = [](auto *kern) {
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, FLUX_WARPS * FLUX_SMEM_PER_WARP * 8);
    };
    flux(k_flux<double, void>);
    flux(k_flux<double, double>);
    flux(k_flux<double, float>);
    flux(k_flux<float, float>);
    cudaFuncSetAttribute(k_sweep_levels, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         SWEEP_WARPS * SWEEP_SMEM_BYTES);
    cudaFuncSetAttribute(k_sweep_df, cudaFuncAttributeMaxDynamicSharedMemorySize, DF_WARPS * SWEEP_SMEM_BYTES);
    // the chain blocks need the largest shared-memory carveout
    auto chain = [](auto *kern) {
        cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, CHAIN_SPREAD_SMEM);
    };
    each_chain_kernel([&](auto *kern, auto *group, bool) {
        chain(kern);
        chain(group);
    });
    done[device] = true;
}

void prepare_launches(int device) { set_attributes(device); }

static int chain_sms(int device) { return device_sms(device) - CH_FREE_SMS; }

int chain_slot_capacity(int device) { return 6 * chain_sms(device); }

bool chain_fits(int device, bool group) {
    static std::mutex mu;
    static int known[256][2] = {};                   // 0: not asked yet, 1: no, 2: yes
    if (device < 0 || device >= 256) return false;
    std::lock_guard<std::mutex> lock(mu);
    int &k = known[device][group ? 1 : 0];
    if (k) return k == 2;
    set_attributes(device);
    auto holds = [](auto *kern, int blocks) {
        int per_sm = 0;
        for (int team = 1; team <= CH_WPB; team *= 2) {
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, CH_WPB * 32, chain_smem_bytes(team)) !=
                cudaSuccess) {
                (void)cudaGetLastError();
                return false;
            }
            if (per_sm < blocks) return false;
        }
        return true;
    };
    bool fits = chain_sms(device) >= 1;
    each_chain_kernel([&](auto *kern, auto *grp, bool three) {
        fits = fits && (group ? holds(grp, three ? 3 : 2) : holds(kern, three ? 3 : 2));
    });
    k = fits ? 2 : 1;
    return fits;
}

int chain_budget(int device, int want, int spread, int *wpb) {
    const int max_blocks = chain_sms(device);
    if (max_blocks < 1) return 0;
    *wpb = spread || want <= 4 * max_blocks ? 4 : 8;
    if (*wpb == 8) want = want * 3 / 4;
    int b = (want + *wpb - 1) / *wpb;
    b = b > max_blocks ? max_blocks : (b < 1 ? 1 : b);
    return !spread && want < *wpb ? (want < 1 ? 1 : want) : b * *wpb;
}

int chain_budget_slots(int budget, int wpb, int precision, int spread) {
    if (wpb < 1) return 0;
    const int each = spread || wpb == 8 ? 6 : (precision != MFCFD_PRECISION_FP64 ? 2 : 3);
    return (budget + wpb - 1) / wpb * each;
}

int chain_count(int device, int budget, int want, int width, int spread) {
    if (spread) return budget;
    long c = (2L * want + 5L * width) / 6;
    const int most = 3 * chain_sms(device);          // teams of four the device holds
    if (want <= 2 * width && c > most && 20 * most >= 17 * width) c = most;
    c = c < budget ? c : budget;
    return c < 1 ? 1 : (int)c;
}

// Rows [a, a + rows) of width w between the reference's index order and
// the storage order: scatter puts row i of src (a transfer buffer in index
// order) at storage row perm[a + i] of dst; gather does the reverse.
__global__ void k_rows(const double *src, double *dst, const int32_t *perm, int a, int rows, int w, int scatter) {
    const size_t total = (size_t)rows * w;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
        const size_t i = t / w, c = t - i * w;
        const size_t s = (size_t)perm[a + i];
        if (scatter) dst[s * w + c] = src[t];
        else dst[t] = src[s * w + c];
    }
}

cudaError_t launch_rows(const double *src, double *dst, const int32_t *perm, int a, int rows, int w, bool scatter,
                        cudaStream_t s) {
    const size_t total = (size_t)rows * w;
    int dev = 0;
    cudaGetDevice(&dev);
    size_t blocks = (total + 255) / 256;
    const size_t cap = (size_t)device_sms(dev) * 8;
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    k_rows<<<(int)blocks, 256, 0, s>>>(src, dst, perm, a, rows, w, scatter ? 1 : 0);
    return cudaGetLastError();
}

cudaError_t launch_qgeo(const DevCloud &d, double *qgeo, cudaStream_t s) {
    k_qgeo<<<(d.n + 127) / 128, 128, 0, s>>>(d, qgeo);
    return cudaGetLastError();
}

cudaError_t launch_conserved_q(const DevCloud &d, cudaStream_t s) {
    k_conserved_q<<<(d.n + 127) / 128, 128, 0, s>>>(d);
    return cudaGetLastError();
}

// A launch with an explicit scheduling priority.  The chain sweep must have
// its blocks placed before those of other handles' flux kernels (which never
// wait, so they cannot hold the sweep up for good); the priority travels with
// the launch, so it holds in a captured graph as on a stream.
template <typename... Args, typename... Act>
static cudaError_t launch_prio(void (*kern)(Args...), int grid, int block, size_t smem, cudaStream_t s, bool high,
                               Act &&...args) {
    // least and greatest priority, looked up once (thread-safe initialisation:
    // group runs may launch from several host threads)
    static const std::pair<int, int> prio = [] {
        int lo = 0, hi = 0;
        cudaDeviceGetStreamPriorityRange(&lo, &hi);
        return std::make_pair(lo, hi);
    }();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributePriority;
    attr[0].val.priority = high ? prio.second : prio.first;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, std::forward<Act>(args)...);
}

// The kernel of a chain sweep in its group form or not: f(kernel).
template <typename F>
static void with_chain_kernel(bool axes, bool mixed, bool dense, F f) {
    int k = 0;
    each_chain_kernel([&](auto *kern, auto *group, bool) {
        if (k++ == (axes ? 0 : 3) + (mixed ? 2 : dense ? 1 : 0)) f(kern, group);
    });
}
// Whether a cloud's sweeps may take the kernels of the global axes and the
// alias driver (no point of a cloud without a shared frame takes the paths in
// question).
static bool chain_axes(const DevCloud &d) { return !d.shared_frame || (d.frame0_axes && !d.dg_old); }

cudaError_t launch_chain_group(const ChainGroup &g, const ChainShape &c, int precision, int forward, cudaStream_t s) {
    const int blocks = g.block_start[g.count], smem = chain_smem(c), threads = CH_WPB * 32;
    bool axes = true;
    for (int i = 0; i < g.count; ++i) axes = axes && chain_axes(g.cloud[i]);
    cudaError_t e = cudaSuccess;
    with_chain_kernel(axes, precision != MFCFD_PRECISION_FP64, c.dense != 0, [&](auto *, auto *group) {
        e = launch_prio(group, blocks, threads, smem, s, true, g, forward);
    });
    return e;
}

cudaError_t launch_iteration(const DevCloud &d, int iter_slot, const IterStreams &st, double *U_next,
                             double *q_next, cudaEvent_t *ev, IterPart part) {
    const int n = d.n;
    cudaStream_t s = st.main;
    int dev = 0;
    cudaGetDevice(&dev);
    set_attributes(dev);
    // dataflow grid: about the widest level in warps (more warps only add
    // pollers), within 8 per SM
    const int sms = device_sms(dev);
    int df_warps = d.max_width;
    df_warps = df_warps < 64 ? 64 : (df_warps > sms * 8 ? sms * 8 : df_warps);
    const int df_blocks = (df_warps + DF_WARPS - 1) / DF_WARPS;
    const bool chains = d.sweep_mode == MFCFD_SWEEP_CHAINS;
    const bool mixed = d.precision != MFCFD_PRECISION_FP64;    // FP32 sweeps; chain schedule only
    const bool dc = d.precision == MFCFD_PRECISION_MIXED_DC;   // ... with the FP64 flux residual
    auto sweep = [&](int forward) {
        if (chains) {
            const ChainShape &c = d.ch_shape;
            const int blocks = chain_blocks(d.ch_chains, c), smem = chain_smem(c), threads = CH_WPB * 32;
            // MIXED and MIXED_DC: folded weights
            with_chain_kernel(chain_axes(d), mixed, c.dense != 0, [&](auto *kern, auto *) {
                launch_prio(kern, blocks, threads, smem, s, true, d, forward);
            });
        } else if (d.sweep_mode == MFCFD_SWEEP_LEVELS) {
            k_sweep_levels<<<1, SWEEP_THREADS, SWEEP_WARPS * SWEEP_SMEM_BYTES, s>>>(d, forward);
        } else {
            cudaMemsetAsync(d.sweep_counter + (forward ? 0 : 1), 0, sizeof(int), s);
            k_sweep_df<<<df_blocks, DF_WARPS * 32, DF_WARPS * SWEEP_SMEM_BYTES, s>>>(d, forward);
        }
    };
    auto mark = [&](int i, cudaStream_t on) { if (ev) cudaEventRecord(ev[i], on); };
    const int fblocks = (n + FLUX_WARPS - 1) / FLUX_WARPS;
    if (part != ITER_ALL && !chains) return cudaErrorInvalidValue;
    if (part == ITER_POST) goto post;
    mark(0, s);
    // supersonic copies may read a neighbour's increment from before the
    // sweeps, which k_pending is about to mark
    if (d.dU_old) cudaMemcpyAsync(d.dU_old, d.dUn, sizeof(double) * 5 * (size_t)n, cudaMemcpyDeviceToDevice, s);
    k_qderiv<<<(n + QD_POINTS - 1) / QD_POINTS, QD_THREADS, 0, s>>>(d);
    for (int j = 0; j < d.inner_iterations; ++j) {
        k_qinner<<<(n + 127) / 128, 128, 0, s>>>(d, d.dq, d.dq_tmp);
        cudaMemcpyAsync(d.dq, d.dq_tmp, sizeof(double) * 15 * (size_t)n, cudaMemcpyDeviceToDevice, s);
    }
    mark(1, s);
    if (chains && d.n_g0 > 0) {
        // phase A of the points outside the shared frame, for both sweeps
        const int gb = (int)(((size_t)d.n_g0 * 32 + 127) / 128);
        if (mixed) k_g0<float><<<gb, 128, 0, s>>>(d);
        else k_g0<double><<<gb, 128, 0, s>>>(d);
    }
    if (chains) {
        // before the sweeps, whose teams leave no room beside them (when the
        // teams came, 1.1M points took about 5% longer with the flux residual
        // beside the forward sweep, 62,400 points 1% less)
        const size_t fsm = FLUX_WARPS * FLUX_SMEM_PER_WARP * 8;
        // a smaller grid walks the same order with its warps striding through it
        const int fgrid = d.flux_grid > 0 && d.flux_grid < fblocks ? d.flux_grid : fblocks;
        const int grid = fgrid + (n + FLUX_WARPS * 32 - 1) / (FLUX_WARPS * 32);
        if (dc) launch_prio(k_flux<double, float>, grid, FLUX_WARPS * 32, fsm, s, false, d);
        else if (mixed) launch_prio(k_flux<float, float>, grid, FLUX_WARPS * 32, fsm, s, false, d);
        else launch_prio(k_flux<double, double>, grid, FLUX_WARPS * 32, fsm, s, false, d);
        mark(2, s);
        mark(3, s);
        if (part == ITER_PRE) {
            cudaEventRecord(st.fork, s);
            return cudaGetLastError();
        }
        sweep(1);
        mark(4, s);
    } else {
        k_flux<double, void><<<fblocks, FLUX_WARPS * 32, FLUX_WARPS * FLUX_SMEM_PER_WARP * 8, s>>>(d);
        mark(2, s);
        k_pending<<<sms * 8, 256, 0, s>>>(d);
        k_dinv_gold<<<(n + 127) / 128, 128, 0, s>>>(d);
        mark(3, s);
        sweep(1);
        mark(4, s);
    }
    sweep(0);
    mark(5, s);
post:
    k_update<<<(n + 127) / 128, 128, 0, s>>>(d, U_next, q_next);
    if (d.n_ss > 0) k_update_ss<<<1, 32, 0, s>>>(d, U_next, q_next);
    mark(6, s);
    const int rb = reduction_blocks(d.n_res);
    k_reduce_partial<<<rb, RED_THREADS, 0, s>>>(d);
    k_reduce_final<<<1, 32, 0, s>>>(d, rb, iter_slot);
    mark(7, s);
    return cudaGetLastError();
}

}  // namespace mfcfd
