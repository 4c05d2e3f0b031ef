// Division on the device: divideMaxLength + divideCells (growth.hpp:66-71, 166-426).
//
//   k_div_count    flags l > Ldiv, counts them (last block: n_divide, capacity check,
//                  sets the graph condition that enables the rest)
//   scan           exclusive scan of the flags -> mother ranks in ascending index order
//   k_div_collect  mothers[rank] = i
//   (cell list of the pre-division cells: bbox, counting sort)
//   k_div_first    one block per mother: room to rotate (min distance to every other cell
//                  >= 2 Rcell, minDistToCell, growth.hpp:82-117, over the bins within
//                  reach), then the first try's draws
//   k_div_near     one block per daughter: min distance to the new population; the last
//                  block counts the satisfied mothers and asks for another try
//   up to 9 x { k_div_try, k_div_near }   the reference's retry loop: every try re-draws
//                  every dividing cell; the last try draws no angles
//   k_div_commit   daughter 1 keeps the mother's row, daughter 2 is appended at n + rank;
//                  IDs max_id + 2k + 1, max_id + 2k + 2; lineage appended; the last block
//                  adds n_divide to n
//
// A division has few mothers (usually one to a few per iteration, at most all cells) and
// some hundred candidate cells around each, so the work per mother is spread over a block:
// its threads share the candidates, and the draws of a try run side by side on the lanes
// of one warp.  With one thread per mother and daughter the serial chain of exact
// distances took 274 + 311 us per event in a 20,000-cell colony and the draws 16-23 us.
// Draws: Philox counters (iteration, mother rank, try, slot), slots 0-3 angles,
// 4-5 length fraction, 6-7 mother growth rate, 8-9 daughter growth rate.
#include "abm_kernels.cuh"

namespace abm {

static inline int cdiv_d(long long a, long long b) { return (int)((a + b - 1) / b); }

const int DV_T = 128;
const int DIV_TRIES = 10;

// FLOW_BEGIN (before the first round of the loop graph): mothers or the cell limit make the
// first iteration a slow one
__global__ void k_div_count(const Phys* __restrict__ phys, Ctrl* ctrl, DivideParams dp, int* flags,
                            unsigned long long cond, int use_cond, int flow)
{
    __shared__ int sh_cnt;
    __shared__ bool last;
    if (flow == FLOW_SLOW && loop_idle(ctrl, flow, true))
    {
        if (use_cond && blockIdx.x == 0 && threadIdx.x == 0)
            cudaGraphSetConditional((cudaGraphConditionalHandle)cond, 0u);
        return;
    }
    if (threadIdx.x == 0) sh_cnt = 0;
    __syncthreads();
    const int n = ctrl->n;
    // terminate() at the top of the loop: no division and no step once n reaches the limit
    const bool halt = ctrl->halt_n > 0 && n >= ctrl->halt_n;
    int cnt = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n && !halt; i += gridDim.x * blockDim.x)
    {
        int f = phys[i].l > dp.Ldiv;          // divideMaxLength, growth.hpp:66-71
        flags[i] = f;
        cnt += f;
    }
    if (cnt) atomicAdd(&sh_cnt, cnt);
    __syncthreads();
    if (threadIdx.x == 0)
    {
        if (sh_cnt) atomicAdd(&ctrl->div_count, sh_cnt);
        __threadfence();
        last = atomicAdd(&ctrl->div_blocks, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (last && threadIdx.x == 0)
    {
        __threadfence();
        int total = atomicAdd(&ctrl->div_count, 0);
        ctrl->div_count = 0;
        ctrl->div_blocks = 0u;
        if (total > 0 && n + total > dp.cap_cells)
        {
            atomicOr(&ctrl->status, (int)ST_CELL_OVERFLOW);
            total = 0;
        }
        ctrl->n_divide = total;
        ctrl->halted = halt ? 1 : 0;
        ctrl->div_done = (total == 0);
        ctrl->div_tries = 0;
        if (use_cond) cudaGraphSetConditional((cudaGraphConditionalHandle)cond, total > 0 ? 1u : 0u);
        if (flow == FLOW_BEGIN)
        {
            ctrl->hold = (total > 0 || halt) ? HOLD_START : HOLD_NONE;
            ctrl->n_divide = 0;            // counted again by the slow iteration
        }
    }
}

__global__ void k_div_collect(const Ctrl* ctrl, const int* flags, const int* rank, int* mothers)
{
    const int n = ctrl->n;
    if (ctrl->n_divide == 0) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        if (flags[i]) mothers[rank[i]] = i;
}

// Any other old cell j (skip_mothers: except rows that now hold daughters) within `limit`
// of the query segment?  Distances taken with the query as cell 1.  This thread's share of
// the candidates: every `step`-th from `first` on, along rows of bins that are contiguous in
// the sorted arrays.  A candidate whose |r| exceeds limit plus both reaches (in FP32 with a
// 1e-4 um margin) is farther than `limit` (the bound of the pair build), so the exact
// distance runs for the few that remain.
__device__ __forceinline__ bool old_cells_within(const Geom& q, int self, const Grid& g,
                                                 const int* __restrict__ bin_start,
                                                 const int* __restrict__ sorted_cell,
                                                 const Geom* __restrict__ sorted_geom, const int* __restrict__ flags,
                                                 bool skip_mothers, double limit, int first, int step)
{
    const X3 rq = x3(q.rx, q.ry, q.rz), nq = x3(q.nx, q.ny, q.nz);
    const double reach = limit + q.h + g.max_half_l;
    const float lim = (float)limit + 1e-4f + segment_reach(q.h, q.nx, q.ny, q.nz);
    const int rings = max(1, (int)ceil(reach * g.inv_edge));
    const int bx = min(max((int)floor((q.rx - g.x0) * g.inv_edge), 0), g.nx - 1);
    const int by = min(max((int)floor((q.ry - g.y0) * g.inv_edge), 0), g.ny - 1);
    const int bz = min(max((int)floor((q.rz - g.z0) * g.inv_edge), 0), g.nz - 1);
    const int x_lo = max(bx - rings, 0), x_hi = min(bx + rings, g.nx - 1);
    for (int zz = max(bz - rings, 0); zz <= min(bz + rings, g.nz - 1); ++zz)
        for (int yy = max(by - rings, 0); yy <= min(by + rings, g.ny - 1); ++yy)
        {
            const int row = (zz * g.ny + yy) * g.nx;
            if (row + x_lo >= g.nbins) continue;
            const int end = bin_start[min(row + x_hi, g.nbins - 1) + 1];
            for (int p = bin_start[row + x_lo] + first; p < end; p += step)
            {
                const Geom gj = load_geom(sorted_geom, p);
                const float fx = (float)(gj.rx - q.rx), fy = (float)(gj.ry - q.ry), fz = (float)(gj.rz - q.rz);
                const float L = lim + segment_reach(gj.h, gj.nx, gj.ny, gj.nz);
                if (fx * fx + fy * fy + fz * fz > L * L) continue;
                const int j = sorted_cell[p];
                if (j == self || (skip_mothers && flags[j])) continue;
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
__device__ __forceinline__ void div_draws(const Geom* __restrict__ geom, const Phys* __restrict__ phys,
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
    const Geom m = load_geom(geom, i);
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

// room checks (growth.hpp:215-236) and the first try, one block per mother
__global__ void __launch_bounds__(DV_T) k_div_first(const Geom* __restrict__ geom, const Phys* __restrict__ phys,
                                                   Ctrl* ctrl, DivideParams dp, const Grid* grid,
                                                   const int* bin_start, const int* sorted_cell,
                                                   const Geom* sorted_geom, const int* flags, const int* mothers,
                                                   int* check, int* sat, Geom* d1, Geom* d2, double* dlen,
                                                   double* dgrowth)
{
    const int nd = ctrl->n_divide;
    const int iter = ctrl->iter;
    const Grid g = *grid;
    for (int k = blockIdx.x; k < nd; k += gridDim.x)
    {
        const int i = mothers[k];
        const bool near = old_cells_within(load_geom(geom, i), i, g, bin_start, sorted_cell, sorted_geom, flags, false,
                                           2 * dp.Rcell, threadIdx.x, DV_T);
        const bool crowded = __syncthreads_or(near);
        if (threadIdx.x < 32) div_draws(geom, phys, dp, iter, k, i, 0, !crowded, d1, d2, dlen, dgrowth);
        if (threadIdx.x == 0)
        {
            check[k] = crowded ? 0 : 1;   // growth.hpp:215-226
            sat[k] = crowded ? 1 : 0;     // :231-236
        }
    }
}

// tr_arg: the try (1 .. DIV_TRIES - 1), or -1 for the try after the ctrl->div_tries
// completed ones (the WHILE node of the iteration graph); one warp per mother
__global__ void __launch_bounds__(DV_T) k_div_try(const Geom* __restrict__ geom, const Phys* __restrict__ phys,
                                                 Ctrl* ctrl, DivideParams dp, const int* mothers, const int* check,
                                                 int tr_arg, Geom* d1, Geom* d2, double* dlen, double* dgrowth)
{
    const int nd = ctrl->n_divide;
    const int tr = tr_arg >= 0 ? tr_arg : ctrl->div_tries;
    if (nd == 0 || ctrl->div_done) return;
    const int iter = ctrl->iter;
    for (int k = (blockIdx.x * DV_T + threadIdx.x) >> 5; k < nd; k += gridDim.x * (DV_T / 32))
        div_draws(geom, phys, dp, iter, k, mothers[k], tr, tr < DIV_TRIES - 1 && check[k] == 1, d1, d2, dlen, dgrowth);
}

// Min distance of each daughter to the new population >= 2 Rcell (growth.hpp:366-398), one
// block per daughter; then the last block marks the satisfied mothers and counts them.
// use_cond: `cond` is the handle of the WHILE node around the further tries, run while a
// dividing cell still misses the distance criterion and tries are left.
__global__ void __launch_bounds__(DV_T) k_div_near(Ctrl* ctrl, DivideParams dp, const Grid* grid,
                                                  const int* bin_start, const int* sorted_cell,
                                                  const Geom* sorted_geom, const int* flags, const int* mothers,
                                                  const int* check, int tr_arg, const Geom* d1, const Geom* d2,
                                                  int* ok, int* sat, unsigned long long cond, int use_cond)
{
    __shared__ bool last;
    const int nd = ctrl->n_divide;
    const int tr = tr_arg >= 0 ? tr_arg : ctrl->div_tries;
    if (nd == 0 || (tr > 0 && ctrl->div_done))
    {
        if (use_cond && blockIdx.x == 0 && threadIdx.x == 0)
            cudaGraphSetConditional((cudaGraphConditionalHandle)cond, 0u);
        return;
    }
    const Grid g = *grid;
    const double limit = 2 * dp.Rcell;
    for (int q = blockIdx.x; q < 2 * nd; q += gridDim.x)
    {
        const int k = q >> 1, which = q & 1;
        bool close = false;
        if (check[k] == 1)
        {
            const Geom dq = which ? d2[k] : d1[k];
            close = old_cells_within(dq, mothers[k], g, bin_start, sorted_cell, sorted_geom, flags, true, limit,
                                     threadIdx.x, DV_T);
            const X3 rq = x3(dq.rx, dq.ry, dq.rz), nq = x3(dq.nx, dq.ny, dq.nz);
            const float lim = (float)limit + 1e-4f + segment_reach(dq.h, dq.nx, dq.ny, dq.nz);
            for (int o = threadIdx.x; o < 2 * nd && !close; o += DV_T)
            {
                if (o == q) continue;
                const Geom go = (o & 1) ? d2[o >> 1] : d1[o >> 1];
                const float fx = (float)(go.rx - dq.rx), fy = (float)(go.ry - dq.ry), fz = (float)(go.rz - dq.rz);
                const float L = lim + segment_reach(go.h, go.nx, go.ny, go.nz);
                if (fx * fx + fy * fy + fz * fz > L * L) continue;
                Dist d = dist_between_cells(rq, nq, dq.h, x3(go.rx, go.ry, go.rz), x3(go.nx, go.ny, go.nz), go.h);
                if (xnorm(x3(d.dx, d.dy, d.dz)) < limit) close = true;
            }
        }
        close = __syncthreads_or(close);
        if (threadIdx.x == 0) ok[q] = (check[k] == 1 && !close) ? 1 : 0;
    }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        __threadfence();
        last = atomicAdd(&ctrl->div_blocks, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    int c = 0;
    for (int k = threadIdx.x; k < nd; k += DV_T)
    {
        if (check[k] == 1 && __ldcg(ok + 2 * k) && __ldcg(ok + 2 * k + 1)) sat[k] = 1;
        c += sat[k];
    }
    // total over the block: counts of the set bits, one per mother and thread round
    __shared__ int sh;
    if (threadIdx.x == 0) sh = 0;
    __syncthreads();
    if (c) atomicAdd(&sh, c);
    __syncthreads();
    if (threadIdx.x == 0)
    {
        ctrl->div_blocks = 0u;
        ctrl->div_tries = tr + 1;
        // while (ntries == 0 || (ntries < 10 && satisfied < n_divide))  (growth.hpp:252)
        ctrl->div_done = (sh >= nd) || (tr + 1 >= DIV_TRIES);
        if (use_cond) cudaGraphSetConditional((cudaGraphConditionalHandle)cond, ctrl->div_done ? 0u : 1u);
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

__global__ void k_div_commit(Geom* geom, Vel* vel, Phys* phys, Ctrl* ctrl, DivideParams dp, const int* mothers,
                             const Geom* d1, const Geom* d2, const double* dlen, const double* dgrowth,
                             int* parents)
{
    __shared__ bool last;
    const int nd = ctrl->n_divide;
    const int n = ctrl->n;
    const int np = ctrl->n_parents;
    const double t = ctrl->t;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nd; k += gridDim.x * blockDim.x)
    {
        const int i = mothers[k];
        const Phys pm = phys[i];
        const Vel vm = vel[i];
        const int parent_id = (int)pm.id;
        const int max_id = np - 1;
        Geom a = d1[k], b = d2[k];
        Phys p1 = pm, p2 = pm;
        p1.l = dlen[2 * k]; p2.l = dlen[2 * k + 1];
        p1.t0 = t; p2.t0 = t;
        p1.growth = dgrowth[2 * k]; p2.growth = dgrowth[2 * k + 1];
        p1.id = max_id + (2 * k + 1); p2.id = max_id + (2 * k + 2);   // growth.hpp:407-418
        if (dp.inherit && n + nd >= dp.n_start_switch) inherit_switch(dp, ctrl->iter, k, p1, p2);
        geom[i] = a; phys[i] = p1;
        geom[n + k] = b; phys[n + k] = p2; vel[n + k] = vm;
        if (dp.feta) dp.feta[n + k] = dp.feta[i];
        parents[np + 2 * k] = parent_id;
        parents[np + 2 * k + 1] = parent_id;
    }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        __threadfence();
        last = atomicAdd(&ctrl->div_blocks, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last || threadIdx.x != 0) return;
    // every block has read the counters: the new population
    ctrl->div_blocks = 0u;
    if (nd == 0) return;
    ctrl->n += nd;
    ctrl->n_parents += 2 * nd;
    ctrl->divisions += nd;
    ctrl->div_events += 1;
    ctrl->last_div_tries = ctrl->div_tries;
    ctrl->n_divide = 0;
    ctrl->screen_valid = 0;            // new cells: the active pair list is stale
}

void launch_div_count(const Phys* phys, Ctrl* ctrl, const DivideParams& dp, int* flags,
                      unsigned long long cond, int use_cond, cudaStream_t st, int flow)
{
    int blocks = max(min(cdiv_d(dp.cap_cells, 256), 296), 1);
    k_div_count<<<blocks, 256, 0, st>>>(phys, ctrl, dp, flags, cond, use_cond, flow);
}

void launch_div_body_pre(Ctrl* ctrl, const int* flags, const int* rank, int* mothers, int cap_cells,
                         cudaStream_t st)
{
    k_div_collect<<<max(cdiv_d(cap_cells, 256), 1), 256, 0, st>>>(ctrl, flags, rank, mothers);
}

// One block per mother or daughter, striding when there are more than fill the chip; a
// capacity of few cells needs no more blocks than it can have mothers.
static int div_blocks(int cap_cells, int per_cell) { return max(min(per_cell * cap_cells, 148 * 8), 1); }

void launch_div_first(const Geom* geom, const Phys* phys, Ctrl* ctrl, const DivideParams& dp, const Grid* grid,
                      const int* bin_start, const int* sorted_cell, const Geom* sorted_geom, const int* flags,
                      const int* mothers, int* check, int* sat, Geom* d1, Geom* d2, double* dlen, double* dgrowth,
                      int* ok, unsigned long long cond, int use_cond, cudaStream_t st)
{
    k_div_first<<<div_blocks(dp.cap_cells, 1), DV_T, 0, st>>>(geom, phys, ctrl, dp, grid, bin_start, sorted_cell,
                                                             sorted_geom, flags, mothers, check, sat, d1, d2, dlen,
                                                             dgrowth);
    k_div_near<<<div_blocks(dp.cap_cells, 2), DV_T, 0, st>>>(ctrl, dp, grid, bin_start, sorted_cell, sorted_geom,
                                                            flags, mothers, check, 0, d1, d2, ok, sat, cond, use_cond);
}

// a further try: of the WHILE node (tr < 0: the try index from ctrl->div_tries), or launched
// in a row (each exits at once when the criterion already holds for every mother)
void launch_div_try_round(const Geom* geom, const Phys* phys, Ctrl* ctrl, const DivideParams& dp, const Grid* grid,
                          const int* bin_start, const int* sorted_cell, const Geom* sorted_geom, const int* flags,
                          const int* mothers, const int* check, int* sat, Geom* d1, Geom* d2, double* dlen,
                          double* dgrowth, int* ok, int tr, unsigned long long cond, int use_cond, cudaStream_t st)
{
    k_div_try<<<div_blocks(cdiv_d(dp.cap_cells, DV_T / 32), 1), DV_T, 0, st>>>(geom, phys, ctrl, dp, mothers, check,
                                                                             tr, d1, d2, dlen, dgrowth);
    k_div_near<<<div_blocks(dp.cap_cells, 2), DV_T, 0, st>>>(ctrl, dp, grid, bin_start, sorted_cell, sorted_geom,
                                                            flags, mothers, check, tr, d1, d2, ok, sat, cond,
                                                            use_cond);
}

int max_division_tries() { return DIV_TRIES; }

void launch_div_commit(Geom* geom, Vel* vel, Phys* phys, Ctrl* ctrl, const DivideParams& dp, const int* mothers,
                       const Geom* d1, const Geom* d2, const double* dlen, const double* dgrowth, int* parents,
                       cudaStream_t st)
{
    k_div_commit<<<max(min(cdiv_d(dp.cap_cells, DV_T), 148 * 8), 1), DV_T, 0, st>>>(geom, vel, phys, ctrl, dp,
                                                                                  mothers, d1, d2, dlen, dgrowth,
                                                                                  parents);
}

}   // namespace abm
