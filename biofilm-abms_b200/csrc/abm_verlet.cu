// Velocity Verlet (integration mode 0: stepVelocityVerlet, mechanics.hpp:2668-2996) with the
// include_constraint force forms.
//   k_pair_pass<..., VERLET>   the pair shares at the current state, over the active pairs
//   k_verlet_cells<0>  forces -> accelerations, half kick, drift of both cell ends
//   k_pair_pass<..., VERLET>   the same at the drifted state (updateNeighborDistances)
//   k_verlet_cells<1>  forces -> accelerations, second half kick, growth; its last block
//                      closes the step
// Both cell passes report how far the cells have moved since the active pairs were listed.
//
// The include_constraint forms (mechanics.hpp:1298-1311, 1554-1566, 1608-1617,
// adhesion.hpp:355-366, mechanics.hpp:718-755, 845-886, 1152-1161): the orientation rows of
// the Hertz, hard-core and friction terms become (s n) x v; those of the JKR term become
// s (v - (n . v) n); the surface terms trade their nz row for x, y torques.  Both are linear
// in the pair's share v and the body coordinate s, so a pair records its share v, s and the
// JKR part of v, and each cell applies n x and the projection to the sums over its row.
// The forces of one half step (mechanics.hpp:2834-2862, 2919-2947): the conservative forces,
// plus the noise, minus the ambient viscosity eta0 l^3 (dr, l^6 (n x dn) / 12)
// (mechanics.hpp:1784-1820), minus the cell-surface friction (mechanics.hpp:1821-1917),
// capped row by row at cell_surface_coulomb_coeff times the constrained surface repulsion.
//
// A cell's serial FP64 chain bounds the cell passes, as it does the Runge-Kutta attempts
// (16 us each for 5,000 cells before, 10 now); the row sums run over the active shares only, cells clear of
// the surface leave its integrals out, and the contact cases are one formula
// (velocity_tilted).
#include "abm_step.cuh"

namespace abm {

const int VV_T = 128;

__device__ __forceinline__ void cross3(const double a[3], const double b[3], double o[3])
{
    o[0] = a[1] * b[2] - a[2] * b[1];
    o[1] = a[2] * b[0] - a[0] * b[2];
    o[2] = a[0] * b[1] - a[1] * b[0];
}

// the generalised force of one half step on cell i at state (g, u); writes f[6]
__device__ __forceinline__ void verlet_force(const StepParams& sp, const VerletArgs& a, int i, const Geom& g,
                                             const Vel& u, const Phys& ph, int iter, double f[6])
{
    const MechParams& P = sp.mp;
    const double n[3] = {g.nx, g.ny, g.nz};
    // the pair sums in CSR order, then the constrained orientation rows
    double F[3] = {0, 0, 0}, Tc[3] = {0, 0, 0}, Tp[3] = {0, 0, 0};
    const int r0 = a.row_ptr[i], na = a.n_act[i];
    for (int k = 0; k < na; k += 2)
    {
        double4 js[2], pp[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) if (k + q < na) { js[q] = a.jbuf[r0 + k + q]; pp[q] = a.pbuf[r0 + k + q]; }
#pragma unroll
        for (int q = 0; q < 2; ++q)
            if (k + q < na)
            {
                const double w = js[q].w;
                F[0] += js[q].x; F[1] += js[q].y; F[2] += js[q].z;
                Tc[0] += w * (js[q].x - pp[q].x); Tc[1] += w * (js[q].y - pp[q].y); Tc[2] += w * (js[q].z - pp[q].z);
                Tp[0] += w * pp[q].x; Tp[1] += w * pp[q].y; Tp[2] += w * pp[q].z;
            }
    }
    double dE[6];
    double tcr[3];
    cross3(n, Tc, tcr);
    const double np = (n[0] * Tp[0] + n[1] * Tp[1]) + n[2] * Tp[2];
    dE[0] = F[0]; dE[1] = F[1]; dE[2] = F[2];
    dE[3] = tcr[0] + (Tp[0] - np * n[0]);
    dE[4] = tcr[1] + (Tp[1] - np * n[1]);
    dE[5] = tcr[2] + (Tp[2] - np * n[2]);
    // cell-surface repulsion and adhesion, include_constraint (mechanics.hpp:673-910), and the
    // area integrals of the friction (integrals.hpp:400-463)
    double rep[6] = {0, 0, 0, 0, 0, 0}, adh[6] = {0, 0, 0, 0, 0, 0};
    double A1 = 0.0, A2 = 0.0, A3 = 0.0;
    const bool a2 = g.nz < P.nz_threshold;
    const double l = ph.l, h = g.h, R = P.R;
    // the test of cell_velocity_fp64: a cell whose lower end is clear of the surface
    const bool clear = P.no_surface || (!a2 && g.rz - h * fabs(g.nz) > R + 1e-6 * (1.0 + fabs(g.rz)));
    if (!clear)
    {
        if (a2) surface_dEdq_flat(P, g.rz, l, ph.sigma0, rep[2], adh[2]);
        else
        {
            const double nz = g.nz, nz2 = nz * nz, onz = 1.0 - nz2;
            const double Rmrz = R - g.rz, inz = 1.0 / nz, ss = Rmrz / nz;
            const bool both = ss > h, any = ss > -h, partial = fabs(ss) < h;
            const double p = any ? Rmrz + h * nz : 0.0, q = both ? Rmrz - h * nz : 0.0;
            const double P1 = sqrt(p), Q1 = sqrt(q);
            const double P3 = P1 * p, Q3 = Q1 * q, P4 = p * p, Q4 = q * q;
            const double P5 = P3 * p, Q5 = Q3 * q, P6 = P4 * p, Q6 = Q4 * q, P7 = P5 * p, Q7 = Q5 * q;
            const double D1 = (P1 - Q1) * inz * 2.0;
            const double D3 = (P3 - Q3) * inz * (2.0 / 3.0);
            const double D4 = (P4 - Q4) * inz * 0.5;
            const double D5 = (P5 - Q5) * inz * (2.0 / 5.0);
            const double D6 = (P6 - Q6) * inz * (2.0 / 6.0);
            const double D7 = (P7 - Q7) * inz * (2.0 / 7.0);
            const double M1 = (D3 - h * (P1 + Q1)) * inz * 2.0;
            const double M3 = (D5 - h * (P3 + Q3)) * inz * (2.0 / 3.0);
            const double M4 = (D6 - h * (P4 + Q4)) * inz * 0.5;
            const double M5 = (D7 - h * (P5 + Q5)) * inz * (2.0 / 5.0);
            const double pf0 = 2 * P.E0;
            rep[2] = -pf0 * (onz * D4 + P.sqrtR * nz2 * D3);
            const double cx = g.ny, cy = -g.nx;
            const double W = onz * M4 + P.sqrtR * nz2 * M3;
            rep[3] = -pf0 * cx * W;
            rep[4] = -pf0 * cy * W;
            const double a0 = P.sqrtR / 2, a1 = 2 * M_PI * R;
            adh[2] = (a0 * onz * D1 + (partial ? (a1 / 2) * nz : 0.0)) * ph.sigma0;
            const double w1 = partial ? (a1 / 2) * ss * nz : 0.0;
            adh[3] = (a0 * onz * M1 - w1) * cx * ph.sigma0;
            adh[4] = (a0 * onz * M1 - w1) * cy * ph.sigma0;
            const double i4 = both ? 2 * h : (any ? ss + h : 0.0);
            const double i5 = (any && !both) ? (ss * ss - h * h) / 2.0 : 0.0;
            const double i6 = both ? 2 * h * h * h / 3.0 : (any ? (ss * ss * ss + h * h * h) / 3.0 : 0.0);
            const double piRnz2 = M_PI * R * nz2;
            A1 = P.sqrtR * onz * D3 + piRnz2 * i4;
            A2 = P.sqrtR * onz * M3 + piRnz2 * i5;
            A3 = P.sqrtR * onz * ((2 * M5 + h * h * (P3 - Q3)) * inz * (2.0 / 3.0)) + piRnz2 * i6;
        }
    }
#pragma unroll
    for (int c = 0; c < 6; ++c) f[c] = ((-dE[c]) - rep[c]) - adh[c];
    if (sp.noise_on)
    {
        // the attempt-0 noise of the iteration (sample_noise of the step), as the
        // Runge-Kutta path draws it
        for (int k = 0; k < 3; ++k)
        {
            uint32_t x[4] = {(uint32_t)iter, 0u, (uint32_t)i, (uint32_t)k};
            philox4x32_10(x, (uint32_t)sp.seed, (uint32_t)(sp.seed >> 32) ^ RNG_PURPOSE_NOISE);
            const double u0 = philox_u01(x[0], x[1]), u1 = philox_u01(x[2], x[3]);
            f[2 * k] += -sp.noise_max[2 * k] + 2 * sp.noise_max[2 * k] * u0;
            f[2 * k + 1] += -sp.noise_max[2 * k + 1] + 2 * sp.noise_max[2 * k + 1] * u1;
        }
    }
    // ambient viscosity (mechanics.hpp:1784-1820)
    const double dn[3] = {u.v[3], u.v[4], u.v[5]};
    double om[3];
    cross3(n, dn, om);
    const double li = l * l * l;
    const double A = ph.eta0 * li, B = ph.eta0 * li * li * li * (1.0 / 12);
    f[0] -= A * u.v[0]; f[1] -= A * u.v[1]; f[2] -= A * u.v[2];
    f[3] -= B * om[0]; f[4] -= B * om[1]; f[5] -= B * om[2];
    if (!clear)
    {
        // cell-surface friction (mechanics.hpp:1821-1917)
        double csf[6] = {0, 0, 0, 0, 0, 0};
        const double q[3] = {u.v[0], u.v[1], 0.0};
        const double m[3] = {om[1] * n[2] - om[2] * n[1], om[2] * n[0] - om[0] * n[2], 0.0};
        const double eta = ph.eta1 * P.invR;
        if (a2)
        {
            const double phz = R - g.rz;
            if (phz > 0)
            {
                const double area = P.sqrtR * sqrt(phz) * l;
                csf[0] = eta * q[0] * area;
                csf[1] = eta * q[1] * area;
                const double cz = n[0] * m[1] - n[1] * m[0];
                csf[5] = eta * cz * area * (l * l) * (1.0 / 12);
            }
        }
        else
        {
            csf[0] = eta * (q[0] * A1 + m[0] * A2);
            csf[1] = eta * (q[1] * A1 + m[1] * A2);
            double c1[3], c2[3];
            cross3(n, q, c1);
            cross3(n, m, c2);
            csf[3] = eta * (c1[0] * A2 + c2[0] * A3);
            csf[4] = eta * (c1[1] * A2 + c2[1] * A3);
            csf[5] = eta * (c1[2] * A2 + c2[2] * A3);
        }
        if (P.coulomb > 0)
        {
            double sf = 0, sr = 0;
            for (int c = 0; c < 6; ++c) { sf += csf[c] * csf[c]; sr += rep[c] * rep[c]; }
            const double fn = sqrt(sf), max_norm = P.coulomb * sqrt(sr);
            if (fn > max_norm)
            {
                const double scale = max_norm / fn;
                for (int c = 0; c < 6; ++c) csf[c] *= scale;
            }
        }
#pragma unroll
        for (int c = 0; c < 6; ++c) f[c] -= csf[c];
    }
}

// accelerations (mechanics.hpp:2863-2877): forces over the mass, the torque split along n
// and across it over the two moments of inertia of a capsule of density rho
__device__ __forceinline__ void verlet_accel(const double f[6], const double n[3], double length, double rho,
                                             double R, double lin[3], double ang[3])
{
    const double volume = M_PI * ((4. / 3.) * (R * R * R) + R * R * length);
    const double mass = rho * volume;
    const double diam = 2 * R, d2 = diam * diam, d3 = d2 * diam, d4 = d3 * diam;
    const double l2 = length * length, l3 = l2 * length;
    const double mom_par = d4 * (length / 32 + diam / 60) * (rho * M_PI);
    const double mom_perp = d2 * (4 * d3 + 15 * length * d2 + 20 * l2 * diam + 10 * l3) / 480 * (rho * M_PI);
    const double im = 1.0 / mass, ipar = 1.0 / mom_par, iperp = 1.0 / mom_perp;
    const double tq[3] = {f[3], f[4], f[5]};
    const double tn = (tq[0] * n[0] + tq[1] * n[1]) + tq[2] * n[2];
    for (int c = 0; c < 3; ++c)
    {
        lin[c] = f[c] * im;
        const double tpar = tn * n[c], tperp = tq[c] - tpar;
        ang[c] = tpar * ipar + tperp * iperp;
    }
}

__device__ __forceinline__ void normalize3(double n[3])
{
    const double nrm = sqrt((n[0] * n[0] + n[1] * n[1]) + n[2] * n[2]);
    n[0] /= nrm; n[1] /= nrm; n[2] /= nrm;
    if (n[2] < 0) { n[0] = -n[0]; n[1] = -n[1]; n[2] = -n[2]; }
}

// the accepted step's bookkeeping (the accepted branch of the controller, with the
// reference's zero error for a Verlet step, simulation.hpp:1786-1798)
__device__ __forceinline__ void verlet_accept(Ctrl* c)
{
    c->attempts += 1;
    c->last_max_error = 0.0;
    const int h = c->hist_pos;
    c->hist_dt[h] = c->dt;
    c->hist_err[h] = 0.0;
    c->hist_acc[h] = 1;
    c->hist_pos = (h + 1) % HIST;
    c->since_div += 1;
    c->cell_steps += c->n;
    c->t += c->dt;
    c->iter += 1;
    c->iterations += 1;
    if (c->dt_write > 0)
    {
        const double t_old_factor = fmod(c->t - c->dt + 1e-12, c->dt_write);
        const double t_new_factor = fmod(c->t + 1e-12, c->dt_write);
        if (t_old_factor > t_new_factor) c->frame_due = 1;
    }
}

template <int PHASE>
__global__ void __launch_bounds__(VV_T) k_verlet_cells(Ctrl* ctrl, StepParams sp, VerletArgs a)
{
    __shared__ double sh_drift[VV_T / 32];
    __shared__ bool last;
    if (ctrl->halted) return;
    const int n = ctrl->n;
    // the grid covers the capacity; blocks past the cells leave at once and are not counted
    const int blocks = max((n + VV_T - 1) / VV_T, 1);
    if (blockIdx.x >= blocks) return;
    const Geom* g_in = PHASE == 0 ? a.geom : a.geom_c;
    const Vel* v_in = PHASE == 0 ? a.vel : a.vel_c;
    Geom* g_out = PHASE == 0 ? a.geom_c : a.geom;
    Vel* v_out = PHASE == 0 ? a.vel_c : a.vel;
    double drift = 0.0;
    const double dt = ctrl->dt, hdt = 0.5 * dt;
    const int iter = ctrl->iter;
    const double R = sp.mp.R;
    const int i = blockIdx.x * VV_T + threadIdx.x;
    if (i < n)
    {
        const Geom g = g_in[i];
        const Vel u = v_in[i];
        const Phys ph = a.phys[i];
        double f[6];
        verlet_force(sp, a, i, g, u, ph, iter, f);
        const double nv[3] = {g.nx, g.ny, g.nz};
        double lin[3], ang[3];
        verlet_accel(f, nv, ph.l, a.rho, R, lin, ang);
        Geom go = g;
        Vel vo;
        if (PHASE == 0)
        {
            // half kick, then the two ends drift with v and the rotation w x (p - q) / 2
            const double dn[3] = {u.v[3], u.v[4], u.v[5]};
            double om[3];
            cross3(nv, dn, om);
            double vi[3], wi[3];
            for (int c = 0; c < 3; ++c) { vi[c] = u.v[c] + hdt * lin[c]; wi[c] = om[c] + hdt * ang[c]; }
            const double r[3] = {g.rx, g.ry, g.rz};
            double p[3], q[3], pq[3];
            for (int c = 0; c < 3; ++c) { p[c] = r[c] - g.h * nv[c]; q[c] = r[c] + g.h * nv[c]; pq[c] = p[c] - q[c]; }
            double cw[3];
            cross3(wi, pq, cw);
            double pn[3], qn[3], rn[3], nn[3];
            for (int c = 0; c < 3; ++c)
            {
                const double half = cw[c] / 2;
                pn[c] = p[c] + dt * (vi[c] + half);
                qn[c] = q[c] + dt * (vi[c] - half);
                rn[c] = (pn[c] + qn[c]) / 2;
                nn[c] = (qn[c] - pn[c]) / ph.l;
            }
            double dni[3];
            cross3(wi, nv, dni);
            normalize3(nn);
            go.rx = rn[0]; go.ry = rn[1]; go.rz = rn[2];
            go.nx = nn[0]; go.ny = nn[1]; go.nz = nn[2];
            for (int c = 0; c < 3; ++c) { vo.v[c] = vi[c]; vo.v[3 + c] = dni[c]; }
            a.whalf[i] = make_double4(wi[0], wi[1], wi[2], 0.0);
        }
        else
        {
            // second half kick at the drifted state, dn = w x n, then growCells
            // (growth.hpp:51-57) with the step's dt
            const double4 wh = a.whalf[i];
            const double wf[3] = {wh.x + hdt * ang[0], wh.y + hdt * ang[1], wh.z + hdt * ang[2]};
            double dni[3];
            cross3(wf, nv, dni);
            for (int c = 0; c < 3; ++c) { vo.v[c] = u.v[c] + hdt * lin[c]; vo.v[3 + c] = dni[c]; }
            double nn[3] = {g.nx, g.ny, g.nz};
            normalize3(nn);
            go.nx = nn[0]; go.ny = nn[1]; go.nz = nn[2];
            const double lg = ph.l + ph.growth * (4 * R / 3 + ph.l) * dt;
            go.h = lg / 2;
            a.phys[i].l = lg;
            if (!(isfinite(go.rx) && isfinite(go.ry) && isfinite(go.rz) && isfinite(nn[0]) && isfinite(nn[1]) &&
                  isfinite(nn[2])))
                atomicOr(&ctrl->status, (int)ST_NAN);
        }
        g_out[i] = go;
        v_out[i] = vo;
        const Geom r = a.gref[i];
        const double ax = go.rx - r.rx, ay = go.ry - r.ry, az = go.rz - r.rz;
        const double bx = go.nx - r.nx, by = go.ny - r.ny, bz = go.nz - r.nz;
        drift = sqrt(ax * ax + ay * ay + az * az) + go.h * sqrt(bx * bx + by * by + bz * bz) + fabs(go.h - r.h);
        // a state that is no number keeps every pair in the list
        if (!isfinite(drift)) drift = 1e300;
    }
    drift = warp_max(drift);
    if ((threadIdx.x & 31) == 0) sh_drift[threadIdx.x >> 5] = drift;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        for (int w = 1; w < VV_T / 32; ++w) drift = fmax(drift, sh_drift[w]);
        if (drift > 0) atomicMax(&ctrl->drift_bits, (unsigned long long)__double_as_longlong(drift));
        __threadfence();
        last = atomicAdd(&ctrl->blocks_done, 1u) == blocks - 1;
    }
    if (threadIdx.x == 0 && last)
    {
        __threadfence();
        ctrl->drift = __longlong_as_double((long long)atomicExch(&ctrl->drift_bits, 0ull));
        ctrl->blocks_done = 0u;
        if (PHASE == 1) verlet_accept(ctrl);
    }
}

void launch_verlet_cells(int phase, const VerletArgs& a, Ctrl* ctrl, const StepParams& sp, int cap_cells,
                         cudaStream_t st)
{
    const int blocks = max((cap_cells + VV_T - 1) / VV_T, 1);
    if (phase == 0) k_verlet_cells<0><<<blocks, VV_T, 0, st>>>(ctrl, sp, a);
    else k_verlet_cells<1><<<blocks, VV_T, 0, st>>>(ctrl, sp, a);
}

}   // namespace abm
