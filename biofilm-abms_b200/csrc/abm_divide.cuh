// Division on the device: divideMaxLength + divideCells (growth.hpp:66-71, 166-426), the
// phases of the cooperative build launch (abm_build.cu):
//   draw     room to rotate (first try: min distance to every other cell >= 2 Rcell,
//            minDistToCell, growth.hpp:82-117, over the bins within reach) and the draws of
//            one try, a block per mother
//   near     min distance of each daughter to the new population, a block per daughter
//   (the reference's retry loop: every try re-draws every dividing cell, up to ten; the
//   last try draws no angles)
//   commit   daughter 1 keeps the mother's row, daughter 2 is appended at n + rank;
//            IDs max_id + 2k + 1, max_id + 2k + 2; lineage appended
// Draws: Philox counters (iteration, mother rank, try, slot), slots 0-3 angles,
// 4-5 length fraction, 6-7 mother growth rate, 8-9 daughter growth rate.
//
// A division has few mothers (usually one to a few per iteration, at most all cells) and
// some hundred candidate cells around each, so the work per mother is spread over a block:
// its threads share the candidates, and the draws of a try run side by side on the lanes
// of one warp.  With one thread per mother and daughter the serial chain of exact
// distances took 274 + 311 us per event in a 20,000-cell colony and the draws 16-23 us.
#pragma once
#include "abm_kernels.cuh"

namespace abm {

const int DIV_TRIES = 10;

// Any other old cell j (skip_mothers: except rows that now hold daughters) within `limit`
// of the query segment?  Distances taken with the query as cell 1.  This thread's share of
// the candidates: the block's warps take the rows of bins in turn (a row is contiguous in the
// sorted arrays), its lanes the cells of a row.  A candidate whose |r| exceeds limit plus both reaches (in FP32 with
// the grid's margin) is farther than `limit` (the bound of the pair search), so the exact
// distance runs for the few that remain.
__device__ __forceinline__ bool old_cells_within(const BuildArgs& a, const Geom& q, int self, const Grid& g,
                                                 bool skip_mothers, double limit)
{
    const int warp = threadIdx.x >> 5, warps = blockDim.x >> 5, lane = threadIdx.x & 31;
    const X3 rq = x3(q.rx, q.ry, q.rz), nq = x3(q.nx, q.ny, q.nz);
    const double reach = limit + q.h + g.max_half_l;
    const float lim = (float)limit + g.margin + segment_reach(q.h, q.nx, q.ny, q.nz);
    const float qx = (float)(q.rx - g.x0), qy = (float)(q.ry - g.y0), qz = (float)(q.rz - g.z0);
    // no more rings than the grid has bins, whatever the longest cell's length: the sums below
    // stay in range
    const int rings = max(1, (int)fmin(ceil(reach * g.inv_edge), (double)max(g.nx, max(g.ny, g.nz))));
    const int bx = min(max((int)floor((q.rx - g.x0) * g.inv_edge), 0), g.nx - 1);
    const int by = min(max((int)floor((q.ry - g.y0) * g.inv_edge), 0), g.ny - 1);
    const int bz = min(max((int)floor((q.rz - g.z0) * g.inv_edge), 0), g.nz - 1);
    const int x_lo = max(bx - rings, 0), x_hi = min(bx + rings, g.nx - 1);
    const int z0 = max(bz - rings, 0), y0 = max(by - rings, 0);
    const int ny = min(by + rings, g.ny - 1) - y0 + 1, rows = (min(bz + rings, g.nz - 1) - z0 + 1) * ny;
    for (int r = warp; r < rows; r += warps)
    {
        const int row = ((z0 + r / ny) * g.ny + y0 + r % ny) * (g.nx + 1);
        const int end = a.bin_start[row + x_hi + 1];
        for (int p = a.bin_start[row + x_lo] + lane; p < end; p += 32)
        {
            const float4 o = a.sorted_pos[p];
            const float fx = o.x - qx, fy = o.y - qy, fz = o.z - qz, L = lim + o.w;
            if (fx * fx + fy * fy + fz * fz > L * L) continue;
            const int j = a.sorted_cell[p];
            if (j == self || (skip_mothers && a.flags[j])) continue;
            const Geom gj = a.geom[j];
            const Dist d = dist_between_cells(rq, nq, q.h, x3(gj.rx, gj.ry, gj.rz), x3(gj.nx, gj.ny, gj.nz), gj.h);
            if (xnorm(x3(d.dx, d.dy, d.dz)) < limit) return true;
        }
    }
    return false;
}

__device__ __forceinline__ double div_u(const DivideParams& dp, int iter, int k, int tr, int slot)
{
    return rng_uniform(dp.seed, RNG_PURPOSE_DIVIDE, (uint32_t)iter, (uint32_t)k, (uint32_t)tr, (uint32_t)slot);
}

// utils.hpp:791-801 (rotateXY) then :814-829 (rotateOutOfXY), in correctly rounded
// operations without FMA so daughters come out bit-identical to the CPU restatement
__device__ __forceinline__ void rotate_daughter(double ux, double uy, double uz, double st, double ct, double s2,
                                                double c2, double& ox, double& oy, double& oz)
{
    double ax = __dadd_rn(__dadd_rn(__dmul_rn(ct, ux), __dmul_rn(-st, uy)), __dmul_rn(0.0, uz));
    double ay = __dadd_rn(__dadd_rn(__dmul_rn(st, ux), __dmul_rn(ct, uy)), __dmul_rn(0.0, uz));
    double az = __dadd_rn(__dadd_rn(__dmul_rn(0.0, ux), __dmul_rn(0.0, uy)), __dmul_rn(1.0, uz));
    // v = a x z, normalised; w = v x a
    double vx = __dsub_rn(__dmul_rn(ay, 1.0), __dmul_rn(az, 0.0));
    double vy = __dsub_rn(__dmul_rn(az, 0.0), __dmul_rn(ax, 1.0));
    double vz = __dsub_rn(__dmul_rn(ax, 0.0), __dmul_rn(ay, 0.0));
    double vn = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(vx, vx), __dmul_rn(vy, vy)), __dmul_rn(vz, vz)));
    vx = __ddiv_rn(vx, vn); vy = __ddiv_rn(vy, vn); vz = __ddiv_rn(vz, vn);
    double wx = __dsub_rn(__dmul_rn(vy, az), __dmul_rn(vz, ay));
    double wy = __dsub_rn(__dmul_rn(vz, ax), __dmul_rn(vx, az));
    double wz = __dsub_rn(__dmul_rn(vx, ay), __dmul_rn(vy, ax));
    ox = __dadd_rn(__dmul_rn(ax, c2), __dmul_rn(wx, s2));
    oy = __dadd_rn(__dmul_rn(ay, c2), __dmul_rn(wy, s2));
    oz = __dadd_rn(__dmul_rn(az, c2), __dmul_rn(wz, s2));
}

// One try's draws for mother k, by one full warp.  Lanes 0-3 take the sine and cosine of
// the two daughters' in-plane and out-of-plane angles, lanes 4-6 the Box-Muller parts of
// the length fraction and of the two growth rates (the same deterministic functions on
// every lane, so their long serial chains run once instead of seven times); then lanes 0
// and 1 place one daughter each.
__device__ __forceinline__ void div_draws(const Geom* geom, const Phys* phys,
                                          const DivideParams& dp, int iter, int k, int i, int tr, bool angles,
                                          Geom* d1, Geom* d2, double* dlen, double* dgrowth)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    double arg = 0.0, u = 1.0;
    if (lane < 4 && angles)
    {
        const double b = (lane & 1) ? dp.angle_z_bound : dp.angle_xy_bound;
        arg = __dadd_rn(-b, __dmul_rn(__dmul_rn(2.0, b), div_u(dp, iter, k, tr, lane)));
    }
    else if (lane >= 4 && lane < 7)
    {
        const int slot = 4 + 2 * (lane - 4);
        u = div_u(dp, iter, k, tr, slot);
        arg = __dmul_rn(6.283185307179586476925286766559005768, div_u(dp, iter, k, tr, slot + 1));
    }
    double sn, cs;
    det_sincos(arg, sn, cs);
    // utils.hpp:648-655 (standardNormal, Box-Muller), as std_normal
    const double nrm = __dmul_rn(__dsqrt_rn(__dmul_rn(-2.0, det_log(u))), cs);
    const int from = 2 * (lane & 1);
    const double st = __shfl_sync(full, sn, from), ct = __shfl_sync(full, cs, from);
    const double s2 = __shfl_sync(full, sn, from + 1), c2 = __shfl_sync(full, cs, from + 1);
    const double norm_len = __shfl_sync(full, nrm, 4), norm_growth = __shfl_sync(full, nrm, 5 + (lane & 1));
    if (lane >= 2) return;
    const Geom m = geom[i];
    const Phys pm = phys[i];
    Geom a = m;
    rotate_daughter(m.nx, m.ny, m.nz, st, ct, s2, c2, a.nx, a.ny, a.nz);
    // growth.hpp:311-348: lengths M (L - 2R), (1 - M)(L - 2R) and centres either side of
    // the division point (correctly rounded operations, as the CPU restatement)
    const double r = __dadd_rn(0.5, __dmul_rn(dp.daughter_length_std, norm_len));
    const double M = r < 0 ? 0.0 : (r > 1 ? 1.0 : r);
    const double Ld = __dsub_rn(pm.l, __dmul_rn(2.0, dp.R));
    const double L1 = __dmul_rn(M, Ld), L2 = __dmul_rn(__dsub_rn(1.0, M), Ld);
    const double dv = __dadd_rn(__dadd_rn(-m.h, L1), dp.R);
    const double Lk = lane ? L2 : L1;
    const double half = __ddiv_rn(Lk, 2.0), del = __dadd_rn(half, dp.R);
    const double f = lane ? __dadd_rn(dv, del) : __dsub_rn(dv, del);
    a.rx = __dadd_rn(m.rx, __dmul_rn(f, a.nx)); a.ry = __dadd_rn(m.ry, __dmul_rn(f, a.ny));
    a.rz = __dadd_rn(m.rz, __dmul_rn(f, a.nz));
    a.h = half;
    (lane ? d2 : d1)[k] = a;
    dlen[2 * k + lane] = Lk;
    // with switching, the distribution of the mother's group (growth.hpp:634-644)
    double gmean = dp.growth_mean, gstd = dp.growth_std;
    if (dp.group_growth)
    {
        const int g0 = (int)pm.group == 1 ? 0 : 1;
        gmean = dp.gmean[g0]; gstd = dp.gstd[g0];
    }
    dgrowth[2 * k + lane] = __dadd_rn(gmean, __dmul_rn(gstd, norm_growth));
}

// Try `tr`: on the first, room checks (growth.hpp:215-236) by a block per mother; then the
// draws.  Runs on the first nb blocks.
__device__ __forceinline__ void div_draw_phase(const BuildArgs& a, const Grid& g, int nd, int nb, int iter, int tr)
{
    for (int k = blockIdx.x; k < nd; k += nb)
    {
        const int i = a.mothers[k];
        int check = 0;
        if (tr == 0)
        {
            const bool near = old_cells_within(a, a.geom[i], i, g, false, 2 * a.dp.Rcell);
            check = __syncthreads_or(near) ? 0 : 1;      // growth.hpp:215-226
            if (threadIdx.x == 0)
            {
                a.check[k] = check;
                a.sat[k] = 1 - check;                    // :231-236
            }
        }
        else check = a.check[k];
        if (threadIdx.x < 32)
            div_draws(a.geom, a.phys, a.dp, iter, k, i, tr, tr < DIV_TRIES - 1 && check == 1, a.d1, a.d2, a.dlen,
                      a.dgrowth);
    }
}

// Min distance of each daughter to the new population >= 2 Rcell (growth.hpp:366-398)
__device__ __forceinline__ void div_near_phase(const BuildArgs& a, const Grid& g, int nd, int nb)
{
    const double limit = 2 * a.dp.Rcell;
    for (int q = blockIdx.x; q < 2 * nd; q += nb)
    {
        const int k = q >> 1, which = q & 1;
        bool close = false;
        if (a.check[k] == 1)
        {
            const Geom dq = which ? a.d2[k] : a.d1[k];
            close = old_cells_within(a, dq, a.mothers[k], g, true, limit);
            const X3 rq = x3(dq.rx, dq.ry, dq.rz), nq = x3(dq.nx, dq.ny, dq.nz);
            const float lim = (float)limit + 1e-4f + segment_reach(dq.h, dq.nx, dq.ny, dq.nz);
            for (int o = threadIdx.x; o < 2 * nd && !close; o += blockDim.x)
            {
                if (o == q) continue;
                const Geom go = (o & 1) ? a.d2[o >> 1] : a.d1[o >> 1];
                const float fx = (float)(go.rx - dq.rx), fy = (float)(go.ry - dq.ry), fz = (float)(go.rz - dq.rz);
                const float L = lim + segment_reach(go.h, go.nx, go.ny, go.nz);
                if (fx * fx + fy * fy + fz * fz > L * L) continue;
                Dist d = dist_between_cells(rq, nq, dq.h, x3(go.rx, go.ry, go.rz), x3(go.nx, go.ny, go.nz), go.h);
                if (xnorm(x3(d.dx, d.dy, d.dz)) < limit) close = true;
            }
        }
        close = __syncthreads_or(close);
        if (threadIdx.x == 0) a.ok[q] = (a.check[k] == 1 && !close) ? 1 : 0;
    }
}

// switch.hpp:97-142 (switchGroupsInherit) for division pair k, the daughters in the
// mother's row (p1) and the appended row (p2), both of the mother's group g: with
// probability 1 - P(g, g), one of the two, chosen by a second uniform, moves to the other
// group and draws that group's growth rate.  Draws: purpose SWITCH, counters (iteration,
// pair, slot 4 / 5 / 6-7).
__device__ __forceinline__ void inherit_switch(const DivideParams& dp, int iter, int k, Phys& p1, Phys& p2)
{
    const int g = (int)p1.group - 1;
    if (g != 0 && g != 1) return;
    auto u = [&](int slot) {
        return rng_uniform(dp.seed, RNG_PURPOSE_SWITCH, (uint32_t)iter, (uint32_t)k, (uint32_t)slot, 0u);
    };
    const double r = u(4);
    double total = dp.rates[g * 2 + g];
    if (!(r > total)) return;
    for (int j = 0; j < 2; ++j)
    {
        if (j == g) continue;
        const double prob = dp.rates[g * 2 + j];
        if (r > total && r < __dadd_rn(total, prob))
        {
            Phys& w = u(5) < 0.5 ? p1 : p2;
            w.group = j + 1;
            w.growth = __dadd_rn(dp.gmean[j], __dmul_rn(dp.gstd[j], std_normal(u(6), u(7))));
            return;
        }
        total = __dadd_rn(total, prob);
    }
}

__device__ __forceinline__ void div_commit_phase(const BuildArgs& a, int n, int nd, int nb, int np, double t, int iter)
{
    const DivideParams& dp = a.dp;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nd; k += nb * blockDim.x)
    {
        const int i = a.mothers[k];
        const Phys pm = a.phys[i];
        const Vel vm = a.vel[i];
        const int parent_id = (int)pm.id;
        const int max_id = np - 1;
        Phys p1 = pm, p2 = pm;
        p1.l = a.dlen[2 * k]; p2.l = a.dlen[2 * k + 1];
        p1.t0 = t; p2.t0 = t;
        p1.growth = a.dgrowth[2 * k]; p2.growth = a.dgrowth[2 * k + 1];
        p1.id = max_id + (2 * k + 1); p2.id = max_id + (2 * k + 2);   // growth.hpp:407-418
        if (dp.inherit && n + nd >= dp.n_start_switch) inherit_switch(dp, iter, k, p1, p2);
        a.geom[i] = a.d1[k]; a.phys[i] = p1;
        a.geom[n + k] = a.d2[k]; a.phys[n + k] = p2; a.vel[n + k] = vm;
        if (dp.feta) dp.feta[n + k] = dp.feta[i];
        a.parents[np + 2 * k] = parent_id;
        a.parents[np + 2 * k + 1] = parent_id;
    }
}

}   // namespace abm
