// The attempt kernel for tableaux of ABM_STAGES stages (2, 4, 6 or 7), with the friction
// trial passes and decision checks; included by one translation unit per stage count.
#include "abm_step.cuh"

namespace abm {

// Does a friction round run?  The first of an attempt's rounds (FR_FIRST in use_cond) runs
// where the pass found candidates and the iteration is alive, a later one where the check
// before it changed a decision (fr_pending).  Both kernels of a round test it themselves: a
// launch that only set the flag took 1.9 us, twice an iteration.
const int FR_FIRST = 4;
__device__ __forceinline__ bool fr_round(const Ctrl* c, int use_cond, int flow)
{
    if (!(use_cond & FR_FIRST)) return c->fr_pending && !c->halted;
    return c->fr_ncand > 0 && !c->halted && !loop_idle(c, flow);
}

// KIND: MODE_TRIAL / MODE_RETRY / MODE_FINAL inside the loop, 3 = API evaluation.
// Without noise the stage-0 velocity k0 = f(y0) is the same for every attempt of an
// iteration (y0 and the pair forces do not change), so the trial stores it in k0buf
// and the retries and the final attempt read it back.
// Learned controller: the trial (the network's proposal) writes its state in place
// and first copies y0 (with l in the gamma slot) and the stored velocity to
// geom_c / vel_c; a proposal that passes the error test closes the step in the
// trial's last block, one that fails continues with retries and a final attempt
// that read y0 back from that copy.
// use_cond bit 0: `cond` is the retry WHILE node's handle; bit 1: `cond_run` is the
// handle of the IF node around the final attempt (0 after a committed proposal).
// B: blocks per SM that the launch bounds ask for.  2- and 4-stage FP64: four (128
// registers), but six (85, some spilled) where all blocks fit the chip at once with six and
// not with four (75,777 to 113,664 cells): HE21 / BS32 steps at 5,000, 60,000, 90,000 and
// 140,000 cells took 28.1 / 34.8, 39.4 / 45.5, 57.2 / 62.5, 76.8 / 86.0 us with four and
// 29.4 / 36.8, 42.5 / 49.5, 51.5 / 62.7, 83.5 / 104 us with six.  Mixed precision and friction:
// six; the friction trial pass, which would spill, three.  6 and 7 stages: no bound (they
// spill below ~130 registers).
// V: 0 FP64; 1 mixed precision; 2 FP64 with cell-cell friction, whose candidate contacts
// add, at each stage whose planar decision differs from the one at y0, the recorded change
// of their shares; 3 the friction trial pass, which runs only the stages of the cells with
// candidate contacts and records their stage states (z, n_z) for the decision check, with
// no other effect.
template <int S, int KIND, bool NOISE, int DIM, int V, int B>
__global__ void __launch_bounds__(AT_T, B) k_attempt(Geom* geom, Vel* vel, Phys* phys, const Gen6* fcc,
                                                 Ctrl* ctrl, StepParams sp, Geom* geom_c, Vel* vel_c,
                                                 Gen6* err_out, Gen6* k0buf, double eval_dt, int eval_attempt,
                                                 unsigned long long cond, int use_cond, PairGather pg,
                                                 unsigned long long cond_run, int flow)
{
    constexpr bool F32 = V == 1, FRIC = V >= 2, DRY = V == 3;
    __shared__ double sh_max[AT_T / 32], sh_drift[AT_T / 32], sh_path[AT_T / 32];
    __shared__ double4 sh_stat[AT_T / 32];
    __shared__ bool last;
    __shared__ Ctrl sc;                 // the last block's copy of the control record
    // the cell of this thread by the attempt order, read beside the control record (the order
    // has an entry for every cell of the capacity)
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int ordered = (KIND != 3 && sp.order && t < sp.order_cap) ? sp.order[t] : t;
    if (DRY && !fr_round(ctrl, use_cond, flow)) return;
    if (KIND != 3 && ctrl->halted)
    {
        // a halted context takes no step: stop an enclosing WHILE node
        if ((use_cond & 1) && (KIND == MODE_TRIAL || KIND == MODE_RETRY) && blockIdx.x == 0 && threadIdx.x == 0)
            cudaGraphSetConditional((cudaGraphConditionalHandle)cond, 0u);
        if ((use_cond & 2) && KIND == MODE_TRIAL && blockIdx.x == 0 && threadIdx.x == 0)
            cudaGraphSetConditional((cudaGraphConditionalHandle)cond_run, 0u);
        return;
    }
    if (KIND == 3 && (ctrl->halted & HALT_LOST)) return;
    if (KIND != 3 && !DRY && loop_idle(ctrl, flow))
    {
        // nothing to resume: stop an enclosing WHILE node
        if ((use_cond & 1) && blockIdx.x == 0 && threadIdx.x == 0)
            cudaGraphSetConditional((cudaGraphConditionalHandle)cond, 0u);
        return;
    }
    const int n = ctrl->n;
    // the grid covers the capacity; blocks past the cells leave at once and are not counted
    const int blocks = max((n + AT_T - 1) / AT_T, 1);
    if (blockIdx.x >= blocks) return;
    const int n_order = (KIND != 3 && sp.order) ? ctrl->n_order : 0;
    const int mode = ctrl->mode;
    const int iter = ctrl->iter;
    // the learned and PI controllers propose (and test) a step every iteration
    const bool trial_ran = sp.propose || (iter % sp.iter_update_stepsize == 0);
    // k0 is shared across attempts only under the reference controller: a passing
    // proposal needs no second attempt, so it does not store k0 or the total pair force
    const bool share_k0 = !NOISE && !sp.propose;
    double dt;
    int attempt;
    bool load_k0 = false, store_k0 = false;
    if (KIND == MODE_TRIAL)
    {
        if (!trial_ran) return;   // no step-size update this iteration: FINAL runs at dt
        dt = ctrl->dt; attempt = 0; store_k0 = share_k0;
    }
    else if (KIND == MODE_RETRY)
    {
        if (mode != MODE_RETRY)
        {
            // no retry pending: make sure an enclosing WHILE node stops
            if ((use_cond & 1) && blockIdx.x == 0 && threadIdx.x == 0)
                cudaGraphSetConditional((cudaGraphConditionalHandle)cond, 0u);
            return;
        }
        dt = ctrl->dt_try; attempt = ctrl->attempt; load_k0 = share_k0;
    }
    else if (KIND == MODE_FINAL)
    {
        dt = (mode == MODE_FINAL) ? ctrl->dt_try : ctrl->dt;
        attempt = (mode == MODE_FINAL) ? ctrl->attempt : 0;
        load_k0 = share_k0 && trial_ran;
    }
    else { dt = eval_dt; attempt = eval_attempt; }
    // the step was closed by a proposal that passed the error test
    if (KIND == MODE_FINAL && mode == MODE_COMMIT) return;
    // a proposal (learned or PI) advances the state in place; the attempts after a failed
    // proposal start from the copy of y0 it kept
    const bool in_place = !DRY && (KIND == MODE_TRIAL) && sp.propose;
    const bool from_backup = (KIND == MODE_RETRY || KIND == MODE_FINAL) && sp.propose;
    if (DRY) store_k0 = false;
    // friction: stages whose planar decisions differ from those at y0 somewhere
    const bool flips = FRIC && ctrl->fr_nflip > 0;

    // the first attempt of an iteration sums the cell's pair shares (pg.fused); under
    // the reference controller the trial writes the total back for the rest, under the
    // proposing ones every attempt sums them
    const bool do_gather = pg.fused &&
                           (KIND == MODE_TRIAL || (KIND == MODE_FINAL && !trial_ran) || sp.propose);
    double local_max = 0.0;
    bool bad = false, longer = false;
    double st_vmax = 0.0, st_v2 = 0.0, st_g = 0.0, st_near = 0.0;
    // motion of each new segment since the last refresh of the active pairs:
    // |dr| + h' |dn| + |dh| (a Hausdorff bound)
    double local_drift = 0.0;
    double local_path = 0.0;        // mixed precision: the motion of this step alone
    // one cell per thread: the grid covers the capacity (attempt_blocks); thread t takes
    // the t-th cell of the attempt order (cells appended after the order was made, in
    // index order).  The body is a do-while(false) block so that `continue` leaves it.
    if (t < n) do
    {
        const int i = t < n_order ? ordered : t;
        if (DRY)
        {
            // only cells with a candidate contact have stage states to report
            bool any = false;
    const int e1 = pg.row_ptr[i] + pg.n_act[i];
            for (int e = pg.row_ptr[i]; e < e1 && !any; ++e) any = (pg.fmask[e] & FR_CAND) != 0;
            if (!any) continue;
        }
        const Geom g = load_geom(from_backup ? geom_c : geom, i);
        int r0 = 0, na = 0;
        if (do_gather) { r0 = pg.row_ptr[i]; na = pg.n_act[i]; }
        const Vel* vprev = (from_backup ? vel_c : vel) + i;
        const double y0[6] = {g.rx, g.ry, g.rz, g.nx, g.ny, g.nz};
        // non-finite coordinates (the reference's DEBUG_CHECK_CELL_COORDINATES_NAN,
        // simulation.hpp:1803-1821): a position alone enters no velocity, so its error
        // norm would stay finite
#pragma unroll
        for (int c = 0; c < 6; ++c) if (!isfinite(y0[c])) bad = true;
        const double l = from_backup ? g.gamma : phys[i].l;
        const double eta0 = phys[i].eta0, eta1 = phys[i].eta1, sigma0 = phys[i].sigma0;
        if (in_place)
        {
            Geom b = g;
            b.gamma = l;
            geom_c[i] = b;
            vel_c[i] = vel[i];
        }
        const bool a2 = y0[5] < sp.mp.nz_threshold;
        Gen6 cc;
        if (do_gather)
        {
            if constexpr (F32) cc = sum_active_shares(reinterpret_cast<const float4*>(pg.jbuf) + r0, na);
            else cc = sum_active_shares(pg.jbuf + r0, na);
            if (KIND == MODE_TRIAL && !sp.propose && !DRY) pg.fcc_w[i] = cc;
        }
        else cc = (KIND == MODE_TRIAL) ? fcc[i] : load_gen6(fcc, i);
        double f0[6];
        double nz2[4] = {0.0, 0.0, 0.0, 0.0};
        if constexpr (DIM == 2)
        {
            if (NOISE) noise_2d(sp, iter, attempt, i, nz2);
        }
        else base_force<NOISE>(sp, cc, iter, attempt, i, f0);
        CellDrag drag;
        if constexpr (DIM == 2) drag = cell_drag_2d(sp, l, eta0, eta1);
        else drag = cell_drag(l, eta0);
        double k[S][6];
        if (load_k0)
        {
            const double2* kp = reinterpret_cast<const double2*>(k0buf + i);
            double2 a = kp[0], b = kp[1], c = kp[2];
            k[0][0] = a.x; k[0][1] = a.y; k[0][2] = b.x; k[0][3] = b.y; k[0][4] = c.x; k[0][5] = c.y;
        }
        else
        {
            if constexpr (DIM == 2) velocity_2d(y0, drag, cc, nz2, k[0]);
            else cell_velocity<F32>(sp.mp, a2, y0, l, g.h, eta0, eta1, sigma0, drag, vprev, f0, k[0]);
            if (store_k0)
            {
                double2* kp = reinterpret_cast<double2*>(k0buf + i);
                kp[0] = make_double2(k[0][0], k[0][1]);
                kp[1] = make_double2(k[0][2], k[0][3]);
                kp[2] = make_double2(k[0][4], k[0][5]);
            }
        }
#pragma unroll
        for (int st = 1; st < S; ++st)
        {
            double y[6];
#pragma unroll
            for (int c = 0; c < 6; ++c)
            {
                double m = 0.0;
#pragma unroll
                for (int j = 0; j < st; ++j) m += k[j][c] * sp.A[st][j];
                y[c] = y0[c] + m * dt;
            }
            normalize_n(y);
            if constexpr (DIM == 2) velocity_2d(y, drag, cc, nz2, k[st]);
            else if constexpr (FRIC)
            {
                if (DRY) pg.ystage[(size_t)st * pg.ystage_ld + i] = make_double2(y[2], y[5]);
                if (flips)
                {
                    double fs[6];
                    friction_stage_force(pg, i, st, f0, fs);
                    cell_velocity<false>(sp.mp, a2, y, l, g.h, eta0, eta1, sigma0, drag, vprev, fs, k[st]);
                }
                else cell_velocity<false>(sp.mp, a2, y, l, g.h, eta0, eta1, sigma0, drag, vprev, f0, k[st]);
            }
            else cell_velocity<F32>(sp.mp, a2, y, l, g.h, eta0, eta1, sigma0, drag, vprev, f0, k[st]);
        }
        if (DRY)
        {
            pg.ystage[i] = make_double2(y0[2], y0[5]);
            continue;
        }
        double vf1[6], d1[6];
#pragma unroll
        for (int c = 0; c < 6; ++c)
        {
            double s1 = 0.0, s2 = 0.0;
#pragma unroll
            for (int st = 0; st < S; ++st) { s1 += k[st][c] * sp.b[st]; s2 += k[st][c] * sp.bs[st]; }
            vf1[c] = s1;
            d1[c] = s1 * dt;
            double err = d1[c] - s2 * dt;
            double scaled = err / (sp.tol * (1.0 + fabs(y0[c])));
            if (!isfinite(scaled)) bad = true;
            local_max = fmax(local_max, scaled);
            if (KIND == 3 && err_out) err_out[i].f[c] = err;
        }
        if (KIND == MODE_FINAL || KIND == 3 || in_place)
        {
            double y1[6];
#pragma unroll
            for (int c = 0; c < 6; ++c) y1[c] = y0[c] + d1[c];
            normalize_n(y1);
            Geom go = g;
            go.rx = y1[0]; go.ry = y1[1]; go.rz = y1[2]; go.nx = y1[3]; go.ny = y1[4]; go.nz = y1[5];
            Vel vo;
#pragma unroll
            for (int c = 0; c < 6; ++c) vo.v[c] = vf1[c];
            if (KIND == MODE_FINAL || in_place)
            {
                // growCells (growth.hpp:51-57) fused with the accepted step
                const double g_rate = phys[i].growth;
                double lg = l + g_rate * (4 * sp.mp.R / 3 + l) * dt;
                go.h = lg / 2;
                longer = sp.div_on && lg > sp.Ldiv;       // divideMaxLength, growth.hpp:66-71
                {
                    const Geom q = load_geom(pg.gref, i);
                    const double ax = go.rx - q.rx, ay = go.ry - q.ry, az = go.rz - q.rz;
                    const double bx = go.nx - q.nx, by = go.ny - q.ny, bz = go.nz - q.nz;
                    local_drift = fmax(local_drift, sqrt(ax * ax + ay * ay + az * az)
                                                        + go.h * sqrt(bx * bx + by * by + bz * bz)
                                                        + fabs(go.h - q.h));
                    if (F32)
                    {
                        const double cx = go.rx - g.rx, cy = go.ry - g.ry, cz = go.rz - g.rz;
                        const double ex = go.nx - g.nx, ey = go.ny - g.ny, ez = go.nz - g.nz;
                        local_path = fmax(local_path, sqrt(cx * cx + cy * cy + cz * cz)
                                                          + go.h * sqrt(ex * ex + ey * ey + ez * ez)
                                                          + fabs(go.h - g.h));
                    }
                }
                if (from_backup) go.gamma = geom[i].gamma;   // the copy holds l in that slot
                phys[i].l = lg;
                geom[i] = go;
                vel[i] = vo;
                if (sp.stats_on)
                {
                    const double v2 = vf1[0] * vf1[0] + vf1[1] * vf1[1] + vf1[2] * vf1[2];
                    st_vmax = fmax(st_vmax, sqrt(v2));
                    st_v2 += v2;
                    st_g += g_rate;
                    st_near += (lg > sp.near_div_length) ? 1.0 : 0.0;
                }
            }
            else
            {
                geom_c[i] = go;
                vel_c[i] = vo;
            }
        }
    } while (false);
    if (DRY) return;
    if ((KIND == MODE_FINAL || in_place) && sp.stats_on)
    {
        // per-block partials of the step-size features, summed in block order later
        st_vmax = warp_max(st_vmax);
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
        {
            st_v2 += __shfl_xor_sync(0xffffffffu, st_v2, off);
            st_g += __shfl_xor_sync(0xffffffffu, st_g, off);
            st_near += __shfl_xor_sync(0xffffffffu, st_near, off);
        }
        if ((threadIdx.x & 31) == 0) sh_stat[threadIdx.x >> 5] = make_double4(st_vmax, st_v2, st_g, st_near);
        __syncthreads();
        if (threadIdx.x == 0)
        {
            double4 a = sh_stat[0];
            for (int w = 1; w < AT_T / 32; ++w)
            {
                const double4 b = sh_stat[w];
                a.x = fmax(a.x, b.x); a.y += b.y; a.z += b.z; a.w += b.w;
            }
            // the last block sums the partials in block order (no contended atomics)
            sp.stat_part[blockIdx.x] = a;
        }
    }
    if (KIND == MODE_FINAL || in_place)
    {
        if (longer) atomicOr(&ctrl->div_any, 1);
        local_drift = warp_max(local_drift);
        if ((threadIdx.x & 31) == 0) sh_drift[threadIdx.x >> 5] = local_drift;
        if (F32)
        {
            local_path = warp_max(local_path);
            if ((threadIdx.x & 31) == 0) sh_path[threadIdx.x >> 5] = local_path;
        }
    }
    // block max of the scaled error, floored at min_error (simulation.hpp:1703)
    local_max = fmax(local_max, sp.min_error);
    if (bad) local_max = __longlong_as_double(0x7ff0000000000000ll);
    local_max = warp_max(local_max);
    if ((threadIdx.x & 31) == 0) sh_max[threadIdx.x >> 5] = local_max;
    // any thread of the block that met a non-finite value reports it
    const int block_bad = __syncthreads_or(bad ? 1 : 0);
    if (threadIdx.x == 0)
    {
        double m = sh_max[0];
        for (int w = 1; w < AT_T / 32; ++w) m = fmax(m, sh_max[w]);
        unsigned long long bits = (unsigned long long)__double_as_longlong(m);
        if (block_bad) atomicOr(&ctrl->status, (int)ST_NAN);
        if (KIND == MODE_FINAL || in_place)
        {
            double dm = sh_drift[0];
            for (int w = 1; w < AT_T / 32; ++w) dm = fmax(dm, sh_drift[w]);
            if (dm > 0) atomicMax(&ctrl->drift_bits, (unsigned long long)__double_as_longlong(dm));
            if (F32)
            {
                double pm = sh_path[0];
                for (int w = 1; w < AT_T / 32; ++w) pm = fmax(pm, sh_path[w]);
                if (pm > 0) atomicMax(&ctrl->path_bits, (unsigned long long)__double_as_longlong(pm));
            }
        }
        if (KIND == 3) { atomicMax(&ctrl->eval_err_bits, bits); last = false; }
        else
        {
            atomicMax(&ctrl->err_bits, bits);
            __threadfence();
            unsigned int done = atomicAdd(&ctrl->blocks_done, 1u);
            last = (done == blocks - 1);
        }
    }
    __syncthreads();
    if (KIND == 3 || !last) return;
    // The last block works on a copy of the control record, fetched and put back by all its
    // threads at once: one field after another, each a trip to L2 behind the store before it,
    // the controller took longer than some cells' velocities.
    __threadfence();
    static_assert(sizeof(Ctrl) % 8 == 0, "the control record is copied in 8-byte words");
    for (int w = threadIdx.x; w < (int)(sizeof(Ctrl) / 8); w += AT_T)
        reinterpret_cast<unsigned long long*>(&sc)[w] = __ldcg(reinterpret_cast<const unsigned long long*>(ctrl) + w);
    __syncthreads();
    if ((KIND == MODE_FINAL || in_place) && sp.stats_on)
    {
        // step-size features of the accepted step (a failed proposal's are replaced
        // by the final attempt's): every block's partial, in block order
        double4 a = make_double4(0.0, 0.0, 0.0, 0.0);
        for (int b = threadIdx.x; b < blocks; b += AT_T)
        {
            const double2* q = reinterpret_cast<const double2*>(sp.stat_part + b);
            const double2 p0 = __ldcg(q), p1 = __ldcg(q + 1);
            a.x = fmax(a.x, p0.x); a.y += p0.y; a.z += p1.x; a.w += p1.y;
        }
        a.x = warp_max(a.x);
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
        {
            a.y += __shfl_xor_sync(0xffffffffu, a.y, off);
            a.z += __shfl_xor_sync(0xffffffffu, a.z, off);
            a.w += __shfl_xor_sync(0xffffffffu, a.w, off);
        }
        __syncthreads();
        if ((threadIdx.x & 31) == 0) sh_stat[threadIdx.x >> 5] = a;
        __syncthreads();
        if (threadIdx.x == 0)
        {
            double4 t = sh_stat[0];
            for (int w = 1; w < AT_T / 32; ++w)
            {
                const double4 b = sh_stat[w];
                t.x = fmax(t.x, b.x); t.y += b.y; t.z += b.z; t.w += b.w;
            }
            sc.st_vmax_bits = (unsigned long long)__double_as_longlong(t.x);
            sc.st_v2_fx = (unsigned long long)llrint(ldexp(t.y, STAT_V2_SHIFT));
            sc.st_g_fx = (unsigned long long)llrint(ldexp(fmax(t.z, 0.0), STAT_G_SHIFT));
            sc.st_near_div = (unsigned long long)t.w;
        }
    }
    if (threadIdx.x == 0)
    {
        const double E = fmax(__longlong_as_double((long long)sc.err_bits), sp.min_error);
        // motion of the new state, counted once the step is accepted
        const double dm = __longlong_as_double((long long)sc.drift_bits);
        const double pm = F32 ? __longlong_as_double((long long)sc.path_bits) : 0.0;
        if (KIND == MODE_FINAL) { sc.drift = dm; sc.path += pm; }
        const bool grown = sc.div_any != 0;
        sc.drift_bits = 0ull;
        sc.path_bits = 0ull;
        sc.err_bits = 0ull;
        sc.blocks_done = 0u;
        sc.div_any = 0;
        controller_finish(&sc, sp, KIND, E, grown);
        if (in_place && sc.mode == MODE_COMMIT)
        {
            // the proposal passed: its state is in place; close the step and leave
            // MODE_COMMIT so that this iteration's final attempt exits at once
            sc.drift = dm;
            sc.path += pm;
            controller_finish(&sc, sp, MODE_FINAL, E, grown, true);
            sc.mode = MODE_COMMIT;
        }
        else if (flow == FLOW_FAST && KIND == MODE_TRIAL && (sp.propose || sc.mode == MODE_RETRY))
            sc.hold = HOLD_RETRY;          // the slow iteration goes on from here
        // another retry?  (bounded: the controller schedules at most max_tries of them)
        if ((use_cond & 1) && (KIND == MODE_TRIAL || KIND == MODE_RETRY))
            cudaGraphSetConditional((cudaGraphConditionalHandle)cond,
                                    (sc.mode == MODE_RETRY && sc.tries < sp.max_tries) ? 1u : 0u);
        if ((use_cond & 2) && KIND == MODE_TRIAL)
            cudaGraphSetConditional((cudaGraphConditionalHandle)cond_run, sc.mode != MODE_COMMIT ? 1u : 0u);
    }
    __syncthreads();
    for (int w = threadIdx.x; w < (int)(sizeof(Ctrl) / 8); w += AT_T)
        reinterpret_cast<unsigned long long*>(ctrl)[w] = reinterpret_cast<const unsigned long long*>(&sc)[w];
}

// Friction decision check over the candidate pairs of the last pair pass: the planar
// decision of each stage from the two cells' stage states (the contact points
// r + s n of both cells below 1.01 R, mechanics.hpp:1090-1110), compared with the one at
// y0; a pair whose set of differing stages changed is updated in both entries.  The last
// block schedules another trial pass when any pair changed.  One thread per candidate; the
// blocks past them leave at once and are not counted, which took this launch from 4.6 to
// 3.2 us (100 iterations of 10,000 cells, with the launch that fr_round saves: 6.17 -> 6.06 ms).
template <int S>
__global__ void k_fr_check(Ctrl* ctrl, const int4* __restrict__ act, const int* __restrict__ fr_list,
                           const double4* __restrict__ jbuf, const double2* __restrict__ ystage, int ld,
                           int* fmask, double R, int use_cond, int flow)
{
    __shared__ bool last;
    const int m = ctrl->fr_ncand;
    const int blocks = min(max((m + (int)blockDim.x - 1) / (int)blockDim.x, 1), (int)gridDim.x);
    if (blockIdx.x >= blocks) return;
    if (!fr_round(ctrl, use_cond, flow))
    {
        // no first round: no later one either
        if (blockIdx.x == 0 && threadIdx.x == 0 && (use_cond & FR_FIRST)) ctrl->fr_pending = 0;
        return;
    }
    const double lim = 1.01 * R;
    int changed = 0, nflip = 0;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < m; q += blocks * blockDim.x)
    {
        const int4 pr = act[fr_list[q]];
        const double s = jbuf[pr.z].w, t = jbuf[pr.w].w;
        const int mk = fmask[pr.z];
        const bool d0 = (mk & FR_D0) != 0;
        int fl = 0;
        for (int st = 1; st < S; ++st)
        {
            const double2 a = ystage[(size_t)st * ld + pr.x], b = ystage[(size_t)st * ld + pr.y];
            const bool flat = __dadd_rn(a.x, __dmul_rn(s, a.y)) < lim && __dadd_rn(b.x, __dmul_rn(t, b.y)) < lim;
            if (flat != d0) fl |= 1 << st;
        }
        if (fl != (mk & FR_FLIPS))
        {
            fmask[pr.z] = (mk & ~FR_FLIPS) | fl;
            fmask[pr.w] = (fmask[pr.w] & ~FR_FLIPS) | fl;
            changed = 1;
        }
        nflip += fl != 0;
    }
    changed = __syncthreads_or(changed);
    if (nflip) atomicAdd(&ctrl->fr_nflip_next, nflip);
    if (threadIdx.x == 0)
    {
        if (changed) atomicOr(&ctrl->fr_changed, 1);
        __threadfence();
        last = atomicAdd(&ctrl->fr_blocks, 1u) == blocks - 1;
    }
    __syncthreads();
    if (last && threadIdx.x == 0)
    {
        __threadfence();
        ctrl->fr_nflip = atomicAdd(&ctrl->fr_nflip_next, 0);
        ctrl->fr_nflip_next = 0;
        ctrl->fr_pending = atomicAdd(&ctrl->fr_changed, 0);
        ctrl->fr_changed = 0;
        ctrl->fr_blocks = 0u;
    }
}

template <int KIND, bool NOISE, int DIM, int V, int B>
static void launch_bound(const AttemptArgs& a, cudaStream_t st)
{
    k_attempt<ABM_STAGES, KIND, NOISE, DIM, V, B><<<attempt_blocks(a.cap_cells), AT_T, 0, st>>>(
        a.geom, a.vel, a.phys, a.fcc, a.ctrl, *a.sp, a.geom_c, a.vel_c, a.err_out, a.k0buf, a.eval_dt, a.eval_attempt,
        a.cond, a.use_cond, a.pg, a.cond_run, a.flow);
}

template <int KIND, bool NOISE, int DIM, int V>
static void launch_one(const AttemptArgs& a, cudaStream_t st)
{
    if constexpr (ABM_STAGES > 4) launch_bound<KIND, NOISE, DIM, V, 1>(a, st);
    else if constexpr (V != 0) launch_bound<KIND, NOISE, DIM, V, (V == 3 ? 3 : 6)>(a, st);
    else
    {
        const int blocks = attempt_blocks(a.cells);
        if (blocks > 4 * a.num_sms && blocks <= 6 * a.num_sms) launch_bound<KIND, NOISE, DIM, V, 6>(a, st);
        else launch_bound<KIND, NOISE, DIM, V, 4>(a, st);
    }
}

template <bool NOISE, int DIM, int V>
static void launch_kind(int kind, const AttemptArgs& a, cudaStream_t st)
{
    switch (kind)
    {
        case MODE_TRIAL: launch_one<MODE_TRIAL, NOISE, DIM, V>(a, st); break;
        case MODE_RETRY: launch_one<MODE_RETRY, NOISE, DIM, V>(a, st); break;
        case MODE_FINAL: launch_one<MODE_FINAL, NOISE, DIM, V>(a, st); break;
        default: launch_one<3, NOISE, DIM, V>(a, st); break;
    }
}

template <int DIM, int V>
static void launch_noise(int kind, const AttemptArgs& a, cudaStream_t st)
{
    if (a.sp->noise_on) launch_kind<true, DIM, V>(kind, a, st);
    else launch_kind<false, DIM, V>(kind, a, st);
}

#define ABM_CAT_(a, b) a##b
#define ABM_CAT(a, b) ABM_CAT_(a, b)

void ABM_CAT(launch_attempt_, ABM_STAGES)(int kind, const AttemptArgs& a, int dims, cudaStream_t st)
{
    if (dims == 2)
    {
#if ABM_STAGES <= 4
        // the 2-D driver integrates with Bogacki-Shampine 3(2) (2D/include/simulation.hpp:217-228);
        // Heun-Euler is kept for comparison runs
        launch_noise<2, 0>(kind, a, st);
#endif
    }
    else if (a.sp->mixed) launch_noise<3, 1>(kind, a, st);
    else if (a.sp->fric) launch_noise<3, 2>(kind, a, st);
    else launch_noise<3, 0>(kind, a, st);
}

void ABM_CAT(launch_friction_rounds_, ABM_STAGES)(int kind, const AttemptArgs& a, const int4* act, const int* fr_list,
                                                  int* fmask, double R, cudaStream_t st)
{
    for (int r = 1; r < ABM_STAGES; ++r)
    {
        AttemptArgs b = a;
        if (r == 1) b.use_cond |= FR_FIRST;
        launch_noise<3, 3>(kind, b, st);
        k_fr_check<ABM_STAGES><<<148 * 2, 256, 0, st>>>(a.ctrl, act, fr_list, a.pg.jbuf, a.pg.ystage, a.pg.ystage_ld,
                                                        fmask, R, b.use_cond, a.flow);
    }
}

}   // namespace abm
