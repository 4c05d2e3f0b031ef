// The RK attempt: per-cell velocities, the step-size controller and the attempt kernel.
//
//   k_attempt<S, KIND, NOISE, DIM, V>   (stepRungeKuttaAdaptive, mechanics.hpp:2406-2612;
//                  all stages of a cell in registers, the error norm reduced in the same
//                  kernel, the step-size controller of simulation.hpp:1690-1769 run by the
//                  last block to finish)
//
// One thread per cell runs every stage in registers.  3-D pair forces are stage-invariant
// (the table is not refreshed between stages and include_constraint = false,
// mechanics.hpp:2064), so each stage needs only the cell's own state, its precomputed pair
// force and the surface terms.  Each stage count is a translation unit of its own
// (abm_attempt_2.cu ...): the kernels are large and compile side by side.
#pragma once
#include "abm_kernels.cuh"

namespace abm {

__device__ __forceinline__ double warp_max(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// The orientation of a stage state, normalised, with n_z >= 0: one division and its exact
// corrections (div_by) in place of three divisions, the same bits
__device__ __forceinline__ void normalize_n(double y[6])
{
    const double nrm = sqrt((y[3] * y[3] + y[4] * y[4]) + y[5] * y[5]), inv = 1.0 / nrm;
    y[3] = div_by(y[3], nrm, inv); y[4] = div_by(y[4], nrm, inv); y[5] = div_by(y[5], nrm, inv);
    if (y[5] < 0) { y[3] = -y[3]; y[4] = -y[4]; y[5] = -y[5]; }
}

// Mixed precision: a cell in surface contact (and not lying on the substrate) takes the
// FP32 contact branch (velocity_contact_f32); the others keep the FP64 branches (i) and
// (ii), whose surface forces are zero off the surface and the horizontal shortcut on it.
// The free branch keeps its divisions (velocity_free_or_flat): the compiler contracts the
// FP32 sums of velocity_contact_f32 (a b + c d into one of its two fused forms) by the shape
// of the code around them, and with div_by there a last FP32 bit changed in one contact cell
// of three; the learned controller rounds its features to BF16, so such a bit can change the
// steps of a whole run.
__device__ __forceinline__ void cell_velocity_f32(const MechParams& P, bool a2, const double y[6], double l, double h,
                                                  double eta0, double eta1, double sigma0, const CellDrag& d,
                                                  const Vel* __restrict__ drp, const double f0[6], double v[6])
{
    const bool contacting = surface_contact(P, a2, y, h);
    if (!P.no_surface && contacting && !a2)
    {
        velocity_contact_f32(P, y, l, h, eta0, eta1, sigma0, drp, f0, v);
        return;
    }
    double f[6];
#pragma unroll
    for (int c = 0; c < 6; ++c) f[c] = f0[c];
    if (!P.no_surface && a2)
    {
        double rep2 = 0, adh2 = 0;
        surface_dEdq_flat(P, y[2], l, sigma0, rep2, adh2);
        f[2] = (f[2] - rep2) - adh2;
    }
    velocity_free_or_flat(P, contacting, y, l, eta0, eta1, drp, f, v);
}

template <bool F32>
__device__ __forceinline__ void cell_velocity(const MechParams& P, bool a2, const double y[6], double l, double h,
                                              double eta0, double eta1, double sigma0, CellDrag& d,
                                              const Vel* __restrict__ drp, const double f0[6], double v[6])
{
    if constexpr (F32) cell_velocity_f32(P, a2, y, l, h, eta0, eta1, sigma0, d, drp, f0, v);
    else cell_velocity_fp64(P, a2, y, l, h, eta0, eta1, sigma0, d, drp, f0, v);
}

// -dE/dq of the pair forces (getConservativeForces, mechanics.hpp:1768) plus the
// attempt's noise (mechanics.hpp:2489-2510, forces += noise at :2066)
template <bool NOISE>
__device__ __forceinline__ void base_force(const StepParams& sp, const Gen6& cc, int iter, int attempt, int i,
                                           double f0[6])
{
#pragma unroll
    for (int c = 0; c < 6; ++c) f0[c] = -cc.f[c];
    if (NOISE)
    {
        for (int k = 0; k < 3; ++k)
        {
            uint32_t x[4] = {(uint32_t)iter, (uint32_t)attempt, (uint32_t)i, (uint32_t)k};
            philox4x32_10(x, (uint32_t)sp.seed, (uint32_t)(sp.seed >> 32) ^ RNG_PURPOSE_NOISE);
            double u0 = philox_u01(x[0], x[1]), u1 = philox_u01(x[2], x[3]);
            f0[2 * k] += -sp.noise_max[2 * k] + 2 * sp.noise_max[2 * k] * u0;
            f0[2 * k + 1] += -sp.noise_max[2 * k + 1] + 2 * sp.noise_max[2 * k + 1] * u1;
        }
    }
}

// 2-D noise of one attempt (2D/include/mechanics.hpp:1760-1771): uniform on
// [-max, max] for (rx, ry, nx, ny), from the 3-D counter slots 0, 1, 3, 4
__device__ __forceinline__ void noise_2d(const StepParams& sp, int iter, int attempt, int i, double nz[4])
{
    double u[6];
    for (int k = 0; k < 3; ++k)
    {
        uint32_t x[4] = {(uint32_t)iter, (uint32_t)attempt, (uint32_t)i, (uint32_t)k};
        philox4x32_10(x, (uint32_t)sp.seed, (uint32_t)(sp.seed >> 32) ^ RNG_PURPOSE_NOISE);
        u[2 * k] = philox_u01(x[0], x[1]);
        u[2 * k + 1] = philox_u01(x[2], x[3]);
    }
    const double m = sp.max_noise_2d;
    nz[0] = -m + 2 * m * u[0]; nz[1] = -m + 2 * m * u[1];
    nz[2] = -m + 2 * m * u[3]; nz[3] = -m + 2 * m * u[4];
}

// 2-D getVelocities (2D/include/mechanics.hpp:1503-1667) at stage orientation (y3, y4):
// dE/dq = (F, S - (n . S) n) + noise from the pair sums cc = (F, S); v = -dE/dq / (K, L)
// with K = l (eta0 + eta1 rho_c / R), L = l^3 (...) / 12 (:264-279), as reciprocals in d
__device__ __forceinline__ CellDrag cell_drag_2d(const StepParams& sp, double l, double eta0, double eta1)
{
    CellDrag d;
    const double drag = eta0 + eta1 * sp.rho_c / sp.mp.R;
    d.K = l * drag;
    d.L = l * l * l * drag / 12;
    d.iK = 1.0 / d.K;
    d.iL = 1.0 / d.L;
    d.drxy = d.dnxy = -1.0;
    return d;
}
__device__ __forceinline__ void velocity_2d(const double y[6], const CellDrag& d, const Gen6& cc, const double nz[4],
                                            double v[6])
{
    const double w = y[3] * cc.f[3] + y[4] * cc.f[4];
    const double d0 = cc.f[0] + nz[0], d1 = cc.f[1] + nz[1];
    const double d2 = (cc.f[3] - w * y[3]) + nz[2], d3 = (cc.f[4] - w * y[4]) + nz[3];
    v[0] = div_by(-d0, d.K, d.iK); v[1] = div_by(-d1, d.K, d.iK); v[2] = 0.0;
    v[3] = div_by(-d2, d.L, d.iL); v[4] = div_by(-d3, d.L, d.iL); v[5] = 0.0;
}

__device__ __forceinline__ Gen6 load_gen6(const Gen6* __restrict__ g, int i)
{
    const double2* p = reinterpret_cast<const double2*>(g + i);
    double2 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
    Gen6 o;
    o.f[0] = a.x; o.f[1] = a.y; o.f[2] = b.x; o.f[3] = b.y; o.f[4] = c.x; o.f[5] = c.y;
    return o;
}

__device__ __forceinline__ double4 widen(const double4& v) { return v; }
__device__ __forceinline__ double4 widen(const float4& v)
{
    return make_double4((double)v.x, (double)v.y, (double)v.z, (double)v.w);
}

// dE/dq of a cell from its active shares (v, w): sum v and sum w v, in CSR order (the
// partner's share of a pair carries the minus sign of its force).  Shares are double4, or
// float4 (mixed precision), summed in FP64 either way.  Four loads are in flight at once:
// one load per entry left its whole latency exposed on every entry of the row.
template <class SHARE>
__device__ __forceinline__ Gen6 sum_active_shares(const SHARE* row, int n)
{
    Gen6 f;
#pragma unroll
    for (int c = 0; c < 6; ++c) f.f[c] = 0.0;
    for (int k = 0; k < n; k += 4)
    {
        SHARE s[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) if (k + u < n) s[u] = row[k + u];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (k + u < n)
            {
                const double4 js = widen(s[u]);
                f.f[0] += js.x; f.f[1] += js.y; f.f[2] += js.z;
                f.f[3] += js.w * js.x; f.f[4] += js.w * js.y; f.f[5] += js.w * js.z;
            }
    }
    return f;
}

// Step-size controller, run once per attempt by the last block
// (simulation.hpp:1690-1769; the final re-run is accepted unconditionally).
// commit: the final step copies an accepted proposal (no RK evaluation of its own)
// longer: the step left a cell longer than Ldiv
static __device__ void controller_finish(Ctrl* c, const StepParams& sp, int kind, double E, bool longer,
                                         bool commit = false)
{
    if (!commit) c->attempts += 1;
    if (kind == MODE_TRIAL)
    {
        c->last_trial_error = E;
        bool exceeded = E > 1.0;
        c->first_passed = !exceeded;
        if (exceeded) c->rejected += 1;
        if (sp.log_cap > 0)
        {
            // complete the feature row of this iteration: the log ratio of the largest
            // dt the error model accepts, and of this attempt's dt, to the last accepted dt
            float* row = sp.log_buf + (size_t)(c->log_rows % sp.log_cap) * MLP_LOG_COLS;
            row[32] = (float)(-sp.inv_q1 * log(E));
            row[33] = (float)log(c->dt / c->dt_prev);
            row[34] = (float)log10(E);
            row[35] = exceeded ? 0.f : 1.f;
            c->log_rows += 1;
        }
        if (sp.propose && !exceeded)
        {
            // the proposal passed the error test: accept its candidate state as is
            c->mode = MODE_COMMIT;
            c->tries = 0;
            c->attempt = 1;
            return;
        }
        double factor = 0.9 * pow(1.0 / E, sp.inv_q1);
        if (factor >= 10) factor = 10;
        else if (factor < 0.2) factor = 0.2;
        c->factor = factor;
        c->tries = 0;
        c->attempt = 1;
        if (exceeded && 0 < sp.max_tries) { c->mode = MODE_RETRY; c->dt_try = c->dt * factor; return; }
    }
    else if (kind == MODE_RETRY)
    {
        c->retries += 1;
        c->attempt += 1;
        bool exceeded = E > 1.0;
        double factor = c->factor * (0.9 * pow(1.0 / E, sp.inv_q1));
        bool brk = false;
        if (factor >= 10) { factor = 10; brk = true; }
        else if (factor < 0.2) { factor = 0.2; brk = true; }
        c->factor = factor;
        if (!brk)
        {
            c->tries += 1;
            if (exceeded && c->tries < sp.max_tries) { c->mode = MODE_RETRY; c->dt_try = c->dt * factor; return; }
        }
    }
    else   // MODE_FINAL (or a committed proposal): accepted
    {
        c->last_max_error = E;
        const int h = c->hist_pos;
        // error of the accepted step before this one (1 before any)
        const int hp = (h + HIST - 1) % HIST;
        const double e_prev = c->hist_dt[hp] > 0 ? c->hist_err[hp] : 1.0;
        const double dt_accepted = c->dt;
        c->hist_dt[h] = c->dt;
        c->hist_err[h] = E;
        c->hist_acc[h] = c->first_passed;
        c->hist_pos = (h + 1) % HIST;
        c->since_div += 1;
        c->cell_steps += c->n;
        c->todo -= 1;
        c->hold = (sp.div_on && (longer || (c->halt_n > 0 && c->n >= c->halt_n))) ? HOLD_START : HOLD_NONE;
        c->t += c->dt;
        c->iter += 1;
        c->iterations += 1;
        // a frame is due when the time has just passed a multiple of dt_write
        // (simulation.hpp:2025-2028)
        if (c->dt_write > 0)
        {
            const double t_old_factor = fmod(c->t - c->dt + 1e-12, c->dt_write);
            const double t_new_factor = fmod(c->t + 1e-12, c->dt_write);
            if (t_old_factor > t_new_factor) c->frame_due = 1;
        }
        if (sp.pi)
        {
            // the PI proposal for the next step: dt 0.9 E^(-0.7/k) E_prev^(0.4/k), k the error
            // order + 1 (Gustafsson's PI rule with the parameters of Hairer & Wanner, Solving
            // ODEs II, sec. IV.2), the factor held to [0.2, 10], dt to [min, max] step size
            double f = 0.9 * pow(1.0 / E, 0.7 * sp.inv_q1) * pow(e_prev, 0.4 * sp.inv_q1);
            if (f >= 10) f = 10;
            else if (f < 0.2) f = 0.2;
            double next = dt_accepted * f;
            if (next < sp.min_stepsize) next = sp.min_stepsize;
            else if (next > sp.max_stepsize) next = sp.max_stepsize;
            c->dt = next;
        }
        c->mode = MODE_TRIAL;
        c->tries = 0;
        c->attempt = 0;
        return;
    }
    // clamp and schedule the final re-run (simulation.hpp:1752-1760)
    double factor = c->factor;
    if (c->dt * factor < sp.min_stepsize) factor = sp.min_stepsize / c->dt;
    else if (c->dt * factor > sp.max_stepsize) factor = sp.max_stepsize / c->dt;
    c->dt *= factor;
    c->dt_try = c->dt;
    c->mode = MODE_FINAL;
}

// friction: the force of cell i at stage st, f0 minus the change of the dE/dq shares of its
// candidate contacts whose planar decision at this stage differs from the one at y0; each
// change enters as the pair sum does
__device__ __forceinline__ void friction_stage_force(const PairGather& pg, int i, int st, const double f0[6],
                                                     double fs[6])
{
    double acc[6] = {0, 0, 0, 0, 0, 0};
    const int r0 = pg.row_ptr[i], r1 = r0 + pg.n_act[i];
    for (int e = r0; e < r1; ++e)
    {
        if (!((pg.fmask[e] >> st) & 1)) continue;
        const double4 dv = pg.fbuf[e];
        const double w = pg.jbuf[e].w;
        acc[0] += dv.x; acc[1] += dv.y; acc[2] += dv.z;
        acc[3] += w * dv.x; acc[4] += w * dv.y; acc[5] += w * dv.z;
    }
#pragma unroll
    for (int c = 0; c < 6; ++c) fs[c] = f0[c] - acc[c];
}

}   // namespace abm
