// CUDA kernels of the B200 mechanics step (sm_100a).
//
//   neighbor set, division   abm_build.cu
//   pair force     k_pair_pass<MIXED, DIM>                              (cellCellInteractionForces,
//                  mechanics.hpp:1209-1659; one record per unordered pair, screened
//                  against an active list with a skin, both shares per pair; the last
//                  block makes the step-size proposal of the learned controller)
//   RK attempt     abm_attempt.cuh
#include <cstdio>
#include "abm_grid.cuh"
#include "abm_pair.cuh"
#include "abm_propose.cuh"
#include "abm_step.cuh"

namespace abm {

static inline int cdiv(long long a, long long b) { return (int)((a + b - 1) / b); }

// ---------------------------------------------------------------------------
// Column-major cell arrays <-> device records
// ---------------------------------------------------------------------------
__global__ void k_cells_from_colmajor(const double* __restrict__ cm, int n, int ncols, int ld,
                                      int has_gamma, Geom* geom, Vel* vel, Phys* phys)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    auto c = [&](int col) { return cm[(size_t)col * ld + i]; };
    Geom g;
    g.rx = c(1); g.ry = c(2); g.rz = c(3); g.h = c(14);
    g.nx = c(4); g.ny = c(5); g.nz = c(6); g.gamma = has_gamma ? c(21) : 0.0;
    geom[i] = g;
    Vel v;
    for (int k = 0; k < 6; ++k) v.v[k] = c(7 + k);
    vel[i] = v;
    Phys p;
    p.l = c(13); p.growth = c(16); p.eta0 = c(17); p.eta1 = c(18); p.sigma0 = c(19);
    p.t0 = c(15); p.id = c(0); p.group = c(20);
    phys[i] = p;
}

__global__ void k_cells_to_colmajor(const Geom* __restrict__ geom, const Vel* __restrict__ vel,
                                    const Phys* __restrict__ phys, int n, int ncols, int ld,
                                    int has_gamma, double* cm)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Geom g = geom[i]; Vel v = vel[i]; Phys p = phys[i];
    auto w = [&](int col, double x) { cm[(size_t)col * ld + i] = x; };
    w(0, p.id); w(1, g.rx); w(2, g.ry); w(3, g.rz); w(4, g.nx); w(5, g.ny); w(6, g.nz);
    for (int k = 0; k < 6; ++k) w(7 + k, v.v[k]);
    w(13, p.l); w(14, g.h); w(15, p.t0); w(16, p.growth); w(17, p.eta0); w(18, p.eta1);
    w(19, p.sigma0); w(20, p.group);
    if (has_gamma && ncols > 21) w(21, g.gamma);
}

__global__ void k_gen6_to_colmajor(const Gen6* __restrict__ g, int n, double* cm)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Gen6 v = g[i];
    for (int k = 0; k < 6; ++k) cm[(size_t)k * n + i] = v.f[k];
}

// 2-D layout (ABM-2d/ABM-2d-cpp/include/indices.hpp:17-41): id, r(2), n(2), dr(2), dn(2),
// l, half_l, t0, growth, eta0, eta1, maxeta1, group; the records hold z = nz = 0 and
// maxeta1 in the sigma0 slot
__global__ void k_cells_from_colmajor_2d(const double* __restrict__ cm, int n, int ld, Geom* geom, Vel* vel,
                                         Phys* phys)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    auto c = [&](int col) { return cm[(size_t)col * ld + i]; };
    Geom g;
    g.rx = c(1); g.ry = c(2); g.rz = 0.0; g.h = c(10);
    g.nx = c(3); g.ny = c(4); g.nz = 0.0; g.gamma = 0.0;
    geom[i] = g;
    Vel v;
    v.v[0] = c(5); v.v[1] = c(6); v.v[2] = 0.0; v.v[3] = c(7); v.v[4] = c(8); v.v[5] = 0.0;
    vel[i] = v;
    Phys p;
    p.l = c(9); p.t0 = c(11); p.growth = c(12); p.eta0 = c(13); p.eta1 = c(14); p.sigma0 = c(15);
    p.id = c(0); p.group = c(16);
    phys[i] = p;
}

__global__ void k_cells_to_colmajor_2d(const Geom* __restrict__ geom, const Vel* __restrict__ vel,
                                       const Phys* __restrict__ phys, int n, int ld, double* cm)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Geom g = geom[i]; Vel v = vel[i]; Phys p = phys[i];
    auto w = [&](int col, double x) { cm[(size_t)col * ld + i] = x; };
    w(0, p.id); w(1, g.rx); w(2, g.ry); w(3, g.nx); w(4, g.ny);
    w(5, v.v[0]); w(6, v.v[1]); w(7, v.v[3]); w(8, v.v[4]);
    w(9, p.l); w(10, g.h); w(11, p.t0); w(12, p.growth); w(13, p.eta0); w(14, p.eta1); w(15, p.sigma0);
    w(16, p.group);
}

void launch_cells_from_colmajor_2d(const double* cm, int n, int ncols, int ld, Geom* geom, Vel* vel, Phys* phys,
                                   cudaStream_t st)
{
    if (n <= 0) return;
    k_cells_from_colmajor_2d<<<cdiv(n, 256), 256, 0, st>>>(cm, n, ld, geom, vel, phys);
}

void launch_cells_to_colmajor_2d(const Geom* geom, const Vel* vel, const Phys* phys, int n, int ncols, int ld,
                                 double* cm, cudaStream_t st)
{
    if (n <= 0) return;
    k_cells_to_colmajor_2d<<<cdiv(n, 256), 256, 0, st>>>(geom, vel, phys, n, ld, cm);
}

void launch_cells_from_colmajor(const double* cm, int n, int ncols, int ld, int has_gamma,
                                Geom* geom, Vel* vel, Phys* phys, cudaStream_t st)
{
    if (n <= 0) return;
    k_cells_from_colmajor<<<cdiv(n, 256), 256, 0, st>>>(cm, n, ncols, ld, has_gamma, geom, vel, phys);
}
void launch_cells_to_colmajor(const Geom* geom, const Vel* vel, const Phys* phys, int n, int ncols,
                              int ld, int has_gamma, double* cm, cudaStream_t st)
{
    if (n <= 0) return;
    k_cells_to_colmajor<<<cdiv(n, 256), 256, 0, st>>>(geom, vel, phys, n, ncols, ld, has_gamma, cm);
}
void launch_gen6_to_colmajor(const Gen6* g, int n, double* cm, cudaStream_t st)
{
    if (n <= 0) return;
    k_gen6_to_colmajor<<<cdiv(n, 256), 256, 0, st>>>(g, n, cm);
}

// ---------------------------------------------------------------------------
// ---------------------------------------------------------------------------
// Exclusive scan (three passes: block sums, one-block scan of the sums,
// block scan + offset).  Up to 4096 * 4096 entries.
// ---------------------------------------------------------------------------
const int SCAN_T = 1024, SCAN_PER = 4, SCAN_TILE = SCAN_T * SCAN_PER;

__device__ __forceinline__ int block_exclusive_scan(int v, int* sh_warp, int& total)
{
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sh_warp[wid] = x;
    __syncthreads();
    if (wid == 0)
    {
        int w = (lane < (int)(blockDim.x >> 5)) ? sh_warp[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            int y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        sh_warp[lane] = w;
    }
    __syncthreads();
    int warp_off = wid > 0 ? sh_warp[wid - 1] : 0;
    total = sh_warp[(blockDim.x >> 5) - 1];
    __syncthreads();
    return warp_off + x - v;
}

__global__ void __launch_bounds__(SCAN_T) k_scan_sums(const int* __restrict__ in, const int* len_p,
                                                      int* block_sums)
{
    __shared__ int sh[32];
    const int len = *len_p;
    long long base = (long long)blockIdx.x * SCAN_TILE + (long long)threadIdx.x * SCAN_PER;
    int s = 0;
#pragma unroll
    for (int k = 0; k < SCAN_PER; ++k) if (base + k < len) s += in[base + k];
    int total;
    block_exclusive_scan(s, sh, total);
    if (threadIdx.x == 0) block_sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(SCAN_T) k_scan_top(int* block_sums, int nblocks)
{
    __shared__ int sh[32];
    int base = threadIdx.x * SCAN_PER;
    int v[SCAN_PER], s = 0;
#pragma unroll
    for (int k = 0; k < SCAN_PER; ++k) { v[k] = (base + k < nblocks) ? block_sums[base + k] : 0; s += v[k]; }
    int total;
    int off = block_exclusive_scan(s, sh, total);
#pragma unroll
    for (int k = 0; k < SCAN_PER; ++k) { if (base + k < nblocks) block_sums[base + k] = off; off += v[k]; }
    if (threadIdx.x == 0) block_sums[nblocks] = total;
}

__global__ void __launch_bounds__(SCAN_T) k_scan_final(const int* __restrict__ in, const int* len_p,
                                                       const int* block_sums, int* out, int nblocks)
{
    __shared__ int sh[32];
    const int len = *len_p;
    long long base = (long long)blockIdx.x * SCAN_TILE + (long long)threadIdx.x * SCAN_PER;
    int v[SCAN_PER], s = 0;
#pragma unroll
    for (int k = 0; k < SCAN_PER; ++k) { v[k] = (base + k < len) ? in[base + k] : 0; s += v[k]; }
    int total;
    int off = block_exclusive_scan(s, sh, total) + block_sums[blockIdx.x];
#pragma unroll
    for (int k = 0; k < SCAN_PER; ++k) { if (base + k < len) out[base + k] = off; off += v[k]; }
    if (blockIdx.x == 0 && threadIdx.x == 0) out[len] = block_sums[nblocks];
}

// Arrays of at most SCAN_SINGLE_MAX entries: one block of SCAN_T threads, each
// summing a run of at most 64 consecutive entries, then writing its run's prefixes.
// One launch instead of three, for the many small scans of replicate batches.
const int SCAN_SINGLE_MAX = 1 << 16;

__global__ void __launch_bounds__(SCAN_T) k_scan_single(const int* __restrict__ in, const int* len_p, int* out)
{
    __shared__ int sh[32];
    const int len = *len_p;
    const int per = (len + SCAN_T - 1) / SCAN_T;
    const int b0 = min(threadIdx.x * per, len), b1 = min(b0 + per, len);
    int s = 0;
    for (int k = b0; k < b1; ++k) s += in[k];
    int total;
    int off = block_exclusive_scan(s, sh, total);
    for (int k = b0; k < b1; ++k) { const int v = in[k]; out[k] = off; off += v; }
    if (threadIdx.x == 0) out[len] = total;
}

size_t scan_block_sums_size(int cap) { return (size_t)cdiv(cap, SCAN_TILE) + 1; }

void launch_scan(const int* in, const int* len, int* out, int* block_sums, int cap, cudaStream_t st)
{
    if (cap <= SCAN_SINGLE_MAX)
    {
        k_scan_single<<<1, SCAN_T, 0, st>>>(in, len, out);
        return;
    }
    int nb = max(cdiv(cap, SCAN_TILE), 1);
    k_scan_sums<<<nb, SCAN_T, 0, st>>>(in, len, block_sums);
    k_scan_top<<<1, SCAN_T, 0, st>>>(block_sums, nb);
    k_scan_final<<<nb, SCAN_T, 0, st>>>(in, len, block_sums, out, nb);
}

// 2-D pair (2D/include/mechanics.hpp:448-547 and :572-670 with
// 2D/include/adhesion.hpp:403-448).  Returns p = cell i's translational dE/dq of the
// pair (Hertz v_ij minus strength * the JKR vector); i's torque share is s p and
// j's is (-p, -t p), projected per RK stage with the stage orientation.
__device__ __forceinline__ PairOut pair_force_2d(const Geom& gi, const Geom& gj, const ForceParams& fp,
                                                 bool adhere)
{
    PairOut out;
    out.touch = false;
    Dist d = dist_geom(gi, gj);
    const double mag = xnorm(x3(d.dx, d.dy, d.dz));
    const double overlap = 2 * fp.R - mag;
    if (!(overlap > 0)) return out;
    const double dirx = d.dx / mag, diry = d.dy / mag;
    double prefactor;
    if (overlap < fp.max_overlap) prefactor = fp.pf2d[0] * pow15(overlap);
    else prefactor = fp.pf2d[1] + fp.pf2d[2] * pow15(overlap - fp.max_overlap);
    double px = prefactor * dirx, py = prefactor * diry;
    if (adhere)
    {
        // overlap > 0 implies dist <= 2R
        const double term = M_PI * fp.R * (2 * fp.R - (mag <= fp.adh_mindist ? fp.adh_mindist : mag));
        px -= fp.adh_strength * (term * dirx);
        py -= fp.adh_strength * (term * diry);
    }
    out.vx = px; out.vy = py; out.vz = 0.0;
    out.s = d.s; out.t = d.t; out.ovl = overlap; out.touch = true;
    return out;
}

// ---------------------------------------------------------------------------
// Screened pair pass over the pair records (one per unordered pair: cell i, its
// partner j < i, the lower CSR entry k and the partner's entry rev[k]; the larger
// index is cell 1, as in the reference's j < i loop).  The screen is a lower
// bound on the centreline distance: for any unit vector a, the gap between the
// projections of the two segments on a,
//     a . (c_j - c_i) - h_i |a . n_i| - h_j |a . n_j|,
// bounds their distance from below.  a is the closest-point direction of a
// single-precision estimate, so the bound is nearly tight, and it is evaluated
// in FP64, so it is rigorous (may_touch).  The exact pair force writes the pair's
// two shares: (v, s) into the lower entry and (v, t) into the partner's entry.
// The first attempt sums a cell's whole row in CSR order.
// ---------------------------------------------------------------------------
const int PS_T = 256, PS_TILE_MAX = 2048;

// One pass per iteration.  A refresh iteration (the active list is stale: after a rebuild,
// an upload or a division, or once some cell has moved by half the skin since the last
// refresh, 2 * drift >= skin) screens every pair with the rigorous bound of may_touch and
// lists those that pass as the new active pairs; then, behind a barrier over the pass's
// blocks, each active pair takes its two share slots (the active entries of a row, in
// column order, at the row's start) and is computed.  The other iterations compute the
// active pairs only.  A pair left out stays beyond 2R until the next refresh (its distance
// can fall by at most 2 * drift < skin), so its force is exactly zero in every force law of
// the reference (all need overlap > 0), and a row sum over the active entries adds the same
// terms in the same order.  Every slot is written by exactly one pair, so the order of the
// active list changes no result.  The last block installs a new list.
//
// drift is the largest motion of a cell's segment from where it lay at the refresh, not
// the sum over the steps of the largest motion in each: in a relaxing 200,000-cell state,
// where some cell moves 0.05 um in almost every step, the sum refreshed in 20-40 % of the
// steps (92 us a pass instead of 36).
// the friction part of a touching pair's shares (FP64): v -= the force on i under the
// decision at the attempt's positions; a candidate also records the change of v when the
// decision flips, and is listed for the stage checks
__device__ __forceinline__ void friction_shares(const Geom& gi, const Geom& gj, const int4& pr, const ForceParams& fp,
                                                const Dist& d, double dist, double4& v)
{
    const int i = pr.x, j = pr.y;
    const X3 dv = x3(d.dx, d.dy, d.dz);
    const Vel ui = fp.vel[i], uj = fp.vel[j];
    const double eta = fmin(fp.feta[i], fp.feta[j]);
    double rv[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) rv[c] = (ui.v[c] + d.s * ui.v[3 + c]) - (uj.v[c] + d.t * uj.v[3 + c]);
    const bool cand = fp.surface && fabs(__ddiv_rn(d.dz, dist)) < 1e-3;
    bool flat0 = false;
    if (cand)
    {
        const double lim = 1.01 * fp.R;
        flat0 = __dadd_rn(gi.rz, __dmul_rn(d.s, gi.nz)) < lim && __dadd_rn(gj.rz, __dmul_rn(d.t, gj.nz)) < lim;
    }
    double f[3];
    friction_force(dv, dist, flat0, rv, eta, fp, f);
    v.x -= f[0]; v.y -= f[1]; v.z -= f[2];
    if (cand)
    {
        double g[3];
        friction_force(dv, dist, !flat0, rv, eta, fp, g);
        const double4 delta = make_double4(-(g[0] - f[0]), -(g[1] - f[1]), -(g[2] - f[2]), 0.0);
        fp.fbuf[pr.z] = delta;
        fp.fbuf[pr.w] = make_double4(-delta.x, -delta.y, -delta.z, 0.0);
        const int m = FR_CAND | (flat0 ? FR_D0 : 0);
        fp.fmask[pr.z] = m;
        fp.fmask[pr.w] = m;
    }
    else
    {
        fp.fmask[pr.z] = 0;
        fp.fmask[pr.w] = 0;
    }
}

// One active pair (pr: i, j, i's slot, j's slot): both shares, the partner's with the minus
// sign of its force, so that a cell adds all its shares alike.
template <bool MIXED, int DIM>
__device__ __forceinline__ void pair_shares(const Geom& gi, const Geom& gj, const int4& pr, bool adhere,
                                            const ForceParams& fp, const double* __restrict__ td,
                                            const double* __restrict__ tr, double4* __restrict__ jbuf, double& ovl_max,
                                            bool& fr_cand, int rounding)
{
    const int k = pr.z, r = pr.w;
    PairOut p;
    if (DIM == 2) p = pair_force_2d(gi, gj, fp, adhere);
    else p = MIXED ? pair_force_fp32(gi, gj, fp, td, tr, rounding) : pair_force_fp64(gi, gj, fp, td, tr);
    if (MIXED)
    {
        // mixed precision: the shares are single-precision forces, stored as such
        float4* fb = reinterpret_cast<float4*>(jbuf);
        float4 own = make_float4(0.f, 0.f, 0.f, 0.f), other = own;
        if (p.touch)
        {
            own = make_float4((float)p.vx, (float)p.vy, (float)p.vz, (float)p.s);
            other = make_float4(-own.x, -own.y, -own.z, (float)p.t);
            ovl_max = fmax(ovl_max, p.ovl);
        }
        fb[k] = own;
        fb[r] = other;
    }
    else
    {
        double4 own = make_double4(0.0, 0.0, 0.0, 0.0);
        double t = 0.0;
        if (p.touch)
        {
            own = make_double4(p.vx, p.vy, p.vz, p.s);
            t = p.t;
            ovl_max = fmax(ovl_max, p.ovl);
            if (DIM == 3 && fp.fric)
            {
                const Dist d = {p.dx, p.dy, p.dz, p.s, p.t};
                friction_shares(gi, gj, pr, fp, d, p.dist, own);
                fr_cand = (fp.fmask[k] & FR_CAND) != 0;
            }
        }
        else if (DIM == 3 && fp.fric)
        {
            fp.fmask[k] = 0;
            fp.fmask[r] = 0;
        }
        jbuf[k] = own;
        jbuf[r] = make_double4(-own.x, -own.y, -own.z, t);
    }
}

// The velocity-Verlet share of one active pair: the pair force v with the body coordinate
// (jbuf) and its JKR part (pbuf, mechanics.hpp:1209-1659 and adhesion.hpp:282-526 with
// include_constraint), friction (mechanics.hpp:1031-1175) from the state's own velocities
// and contact points; the partner's with the minus sign.
__device__ __forceinline__ void verlet_shares(const Geom& gi, const Geom& gj, const int4& pr, const ForceParams& fp,
                                              const double* __restrict__ td, const double* __restrict__ tr,
                                              double4* __restrict__ jbuf, double4* __restrict__ pbuf)
{
    const PairOut p = pair_force_fp64(gi, gj, fp, td, tr);
    double4 own = make_double4(0.0, 0.0, 0.0, 0.0), part = own;
    double t = 0.0;
    if (p.touch)
    {
        own = make_double4(p.vx, p.vy, p.vz, p.s);
        t = p.t;
        const double ux = p.dx / p.dist, uy = p.dy / p.dist, uz = p.dz / p.dist;
        part = make_double4(p.mj * ux, p.mj * uy, p.mj * uz, 0.0);
        if (fp.fric)
        {
            const X3 dv = x3(p.dx, p.dy, p.dz);
            const Vel ui = fp.vel[pr.x], uj = fp.vel[pr.y];
            const double eta = fmin(fp.feta[pr.x], fp.feta[pr.y]);
            double rv[3];
#pragma unroll
            for (int c = 0; c < 3; ++c)
                rv[c] = (ui.v[c] + p.s * ui.v[3 + c]) - (uj.v[c] + p.t * uj.v[3 + c]);
            bool flat = false;
            if (fp.surface && fabs(__ddiv_rn(p.dz, p.dist)) < 1e-3)
            {
                const double lim = 1.01 * fp.R;
                flat = __dadd_rn(gi.rz, __dmul_rn(p.s, gi.nz)) < lim &&
                       __dadd_rn(gj.rz, __dmul_rn(p.t, gj.nz)) < lim;
            }
            double f[3];
            friction_force(dv, p.dist, flat, rv, eta, fp, f);
            own.x -= f[0]; own.y -= f[1]; own.z -= f[2];
        }
    }
    jbuf[pr.z] = own;
    jbuf[pr.w] = make_double4(-own.x, -own.y, -own.z, t);
    pbuf[pr.z] = part;
    pbuf[pr.w] = make_double4(-part.x, -part.y, -part.z, 0.0);
}

// With PROPOSE the pass also makes the iteration's step-size proposal
// (mlp_propose_block). Its features read the previous iteration's overlap maximum
// (st_ovl_bits of the other parity, which no block of this pass writes), so the
// proposal depends on nothing this pass computes: the grid's last block makes it
// while the other blocks stride over the pairs, and its chain of dependent reads
// and three network layers runs beside the pair work instead of after it. A grid of
// one block computes its pairs first and proposes at the end. The proposal is a
// template parameter so that the passes without it carry none of its code, and the
// bound of two resident blocks per SM (at most 128 registers) holds the pair loop's
// occupancy whatever the proposal adds.
template <bool MIXED, int DIM, bool PROPOSE, bool VERLET = false>
__global__ void __launch_bounds__(PS_T, 2) k_pair_pass(const Geom* __restrict__ geom, const int4* __restrict__ pairs,
                                                      Ctrl* ctrl, ForceParams fp, const double* __restrict__ td,
                                                      const double* __restrict__ tr, double4* __restrict__ jbuf,
                                                      int* surv, ActiveList al, StepParams sp,
                                                      const float* __restrict__ mlp_w, int flow)
{
    __shared__ bool last;
    if (ctrl->halted || loop_idle(ctrl, flow)) return;
    const bool split = PROPOSE && gridDim.x > 1;
    const bool proposer = split && blockIdx.x == gridDim.x - 1;
    const int work_blocks = split ? gridDim.x - 1 : gridDim.x;
    auto stale = [&](const int& valid, const double& moved) { return !valid || !(2.0 * moved * (1.0 + 1e-6) + 1e-9 < fp.skin); };
    const bool refresh = stale(ctrl->screen_valid, ctrl->drift);
    const int rounding = MIXED && stale(ctrl->path_valid, ctrl->path) ? ROUND_STALE : ROUND_LIST;
    const int lane = threadIdx.x & 31;
    const int stride = work_blocks * blockDim.x;
    double ovl_max = 0.0;
    if (proposer)
    {
        if (al.cluster && refresh) cluster_barrier();
        mlp_propose_block(ctrl, sp, mlp_w);
    }
    else if (refresh)
    {
        const int n_pairs = ctrl->n_dir >> 1, n = ctrl->n;
        const double limit = 2 * fp.R + fp.skin;
        // warp-uniform rounds, so that every ballot covers all 32 lanes
        for (int base = blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < n_pairs; base += stride)
        {
            const int p = base + lane;
            bool keep = false;
            if (p < n_pairs)
            {
                const int4 pr = pairs[p];           // (i, j, lower entry k, partner entry)
                keep = may_touch(load_geom(geom, pr.x), load_geom(geom, pr.y), limit);
                al.keep[pr.z] = keep;
                al.keep[pr.w] = keep;
            }
            // warp-aggregated append of the active pairs
            const unsigned mask = __ballot_sync(0xffffffffu, keep);
            int pos = 0;
            if (lane == 0 && mask) pos = atomicAdd(&ctrl->n_surv_next, __popc(mask));
            pos = __shfl_sync(0xffffffffu, pos, 0);
            if (keep) surv[pos + __popc(mask & ((1u << lane) - 1u))] = p;
        }
        // with a proposer, its block takes part in a cluster's barrier below
        if (al.cluster) cluster_barrier();
        else if (!grid_barrier(al.bar, work_blocks, ctrl)) return;
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        {
            int cnt = 0;
            for (int e = al.row_ptr[i]; e < al.row_ptr[i + 1]; ++e) cnt += al.keep[e];
            al.n_act[i] = cnt;
            al.gref[i] = load_geom(geom, i);
        }
        const int m = __ldcg(&ctrl->n_surv_next);
        for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < m; q += stride)
        {
            const int4 pr = pairs[surv[q]];
            int4 rec = make_int4(pr.x, pr.y, al.row_ptr[pr.x], al.row_ptr[pr.y]);
            {
                int a = 0, b = 0;
                for (int e = rec.z; e < pr.z; ++e) a += al.keep[e];
                for (int e = rec.w; e < pr.w; ++e) b += al.keep[e];
                rec.z += a;
                rec.w += b;
            }
            const bool adhere = DIM == 2 && fp.adhere[pr.z] != 0;
            al.act[q] = make_int4(rec.x, adhere ? rec.y | ACT_ADHERE : rec.y, rec.z, rec.w);
            bool cand = false;
            if constexpr (VERLET)
                verlet_shares(load_geom(geom, rec.x), load_geom(geom, rec.y), rec, fp, td, tr, jbuf, al.pbuf);
            else
                pair_shares<MIXED, DIM>(load_geom(geom, rec.x), load_geom(geom, rec.y), rec, adhere, fp, td, tr, jbuf,
                                        ovl_max, cand, rounding);
            if (cand) fp.fr_list[atomicAdd(&ctrl->fr_ncand_next, 1)] = q;
        }
    }
    else
    {
        const int m = ctrl->n_surv;
        for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < m; q += stride)
        {
            int4 rec = al.act[q];
            const bool adhere = DIM == 2 && rec.y < 0;
            if (DIM == 2) rec.y &= ~ACT_ADHERE;
            bool cand = false;
            if constexpr (VERLET)
                verlet_shares(load_geom(geom, rec.x), load_geom(geom, rec.y), rec, fp, td, tr, jbuf, al.pbuf);
            else
                pair_shares<MIXED, DIM>(load_geom(geom, rec.x), load_geom(geom, rec.y), rec, adhere, fp, td, tr, jbuf,
                                        ovl_max, cand, rounding);
            if (cand) fp.fr_list[atomicAdd(&ctrl->fr_ncand_next, 1)] = q;
        }
    }
    if (fp.stats && !proposer)
    {
        ovl_max = warp_max(ovl_max);
        if (lane == 0 && ovl_max > 0)
            atomicMax(&ctrl->st_ovl_bits[ctrl->iter & 1], (unsigned long long)__double_as_longlong(ovl_max));
    }
    // the pass leaves nothing to close?  (a count over the blocks would only cost its trips)
    const bool restart = MIXED && rounding == ROUND_STALE;
    if (!refresh && !restart && !(fp.fric && !VERLET) && !(PROPOSE && !split)) return;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        __threadfence();
        last = atomicAdd(&ctrl->surv_blocks, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    if (threadIdx.x == 0)
    {
        __threadfence();
        if (refresh)
        {
            ctrl->n_surv = atomicAdd(&ctrl->n_surv_next, 0);
            ctrl->n_surv_next = 0;
            ctrl->screen_valid = 1;
            ctrl->drift = 0.0;
        }
        if (restart) { ctrl->path = 0.0; ctrl->path_valid = 1; }
        if (fp.fric && !VERLET)
        {
            // the candidates of this pass; no stage has a changed decision yet
            ctrl->fr_ncand = atomicAdd(&ctrl->fr_ncand_next, 0);
            ctrl->fr_ncand_next = 0;
            ctrl->fr_nflip = 0;
        }
        ctrl->surv_blocks = 0u;
    }
    if (PROPOSE && !split)
    {
        __syncthreads();
        mlp_propose_block(ctrl, sp, mlp_w);
    }
}

// A cluster of 16 blocks is more than the portable 8: allowed per kernel, and used only where
// the device can place one.
LaunchShape make_shape(const void* kernel, int block, long long threads, bool cluster, int num_sms, int share)
{
    const int MAX_CLUSTER = 16;
    LaunchShape s;
    const long long want = max((threads + block - 1) / block, 1LL);
    if (cluster)
    {
        int size = 1;
        while (size < MAX_CLUSTER && size < want) size *= 2;
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = size; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3(size); cfg.blockDim = dim3(block); cfg.attrs = at; cfg.numAttrs = 1;
        int fits = 0;
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
            cudaOccupancyMaxActiveClusters(&fits, kernel, &cfg) == cudaSuccess && fits > 0)
        {
            s.blocks = size;
            s.cluster = 1;
            return s;
        }
        cudaGetLastError();
    }
    int occ = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, block, 0);
    // a share of the chip, but no less than the largest cluster
    s.blocks = (int)min(want, (long long)max(num_sms * max(occ, 1) / max(share, 1), min(MAX_CLUSTER, num_sms)));
    return s;
}

cudaError_t launch_shape(const void* kernel, const LaunchShape& shape, int block, void** args, cudaStream_t st)
{
    if (!shape.cluster) return cudaLaunchCooperativeKernel(kernel, dim3(shape.blocks), dim3(block), args, 0, st);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = shape.blocks; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(shape.blocks); cfg.blockDim = dim3(block); cfg.stream = st; cfg.attrs = at; cfg.numAttrs = 1;
    return cudaLaunchKernelExC(&cfg, kernel, args);
}

// total dE/dq of each cell from its active shares (the API paths; the loop's first attempt
// does the same sum itself); no number where the pass before it lost its blocks (HALT_LOST)
__global__ void k_pair_sum_rows(const int* __restrict__ row_ptr, const int* __restrict__ n_act, const Ctrl* ctrl,
                                const double4* __restrict__ jbuf, Gen6* fcc, int f32)
{
    const int n = ctrl->n;
    if (ctrl->halted & HALT_LOST)
    {
        const double nan = __longlong_as_double(0x7ff8000000000000ll);
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
            for (int c = 0; c < 6; ++c) fcc[i].f[c] = nan;
        return;
    }
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        fcc[i] = f32 ? sum_active_shares(reinterpret_cast<const float4*>(jbuf) + row_ptr[i], n_act[i])
                     : sum_active_shares(jbuf + row_ptr[i], n_act[i]);
}

cudaError_t launch_pair_screened(const Geom* geom, Ctrl* ctrl, ForceParams fp, const double* jkr_delta,
                                 const double* jkr_radius, Gen6* fcc, double4* jbuf, int mixed, int max_entries,
                                 int cap_cells, int num_sms, cudaStream_t st, int with_sum, int dims, int tile,
                                 int blocks_per_sm, const int4* pairs, int* surv, ActiveList al, int cells, int share,
                                 const StepParams* sp, const float* mlp_w, int flow)
{
    // sp (the loop's pass): the last block also runs the step-size proposal
    StepParams spv{};
    if (sp) spv = *sp;
    const int propose = (sp && sp->stats_on) ? 1 : 0;
    const bool f32 = mixed && dims != 2;
    const int p = propose ? 1 : 0;
    const void* const fn2[2] = {(const void*)k_pair_pass<false, 2, false>, (const void*)k_pair_pass<false, 2, true>};
    const void* const fn3m[2] = {(const void*)k_pair_pass<true, 3, false>, (const void*)k_pair_pass<true, 3, true>};
    const void* const fn3[2] = {(const void*)k_pair_pass<false, 3, false>, (const void*)k_pair_pass<false, 3, true>};
    const void* fn = al.pbuf ? (const void*)k_pair_pass<false, 3, false, true> : dims == 2 ? fn2[p] : f32 ? fn3m[p] : fn3[p];
    // The blocks stride over the pairs; those of a refresh wait for one another, so the launch
    // is one cluster for a small colony (the rule of the build launch), else a cooperative
    // grid.  By default two threads per cell (1.5 to 2 active pairs a cell): blocks without work
    // still join the barrier and take the room of a batch's other colonies.  With a tile set:
    // at least that many pairs per block, at most the blocks resident at once (blocks_per_sm
    // caps them per SM).
    LaunchShape shape;
    if (tile <= 0 && blocks_per_sm <= 0)
        shape = make_shape(fn, PS_T, 2LL * cells + (p ? PS_T : 0), cells <= PAIR_CLUSTER_CELLS, num_sms,
                           share);
    else
    {
        const int max_pairs = max(max_entries / 2, 1);
        shape = make_shape(fn, PS_T, (long long)PS_T * cdiv(max_pairs, tile <= 0 ? 1024 : min(tile, PS_TILE_MAX)), false,
                           num_sms, share);
        if (blocks_per_sm > 0) shape.blocks = min(shape.blocks, num_sms * blocks_per_sm);
    }
    al.cluster = shape.cluster;
    void* args[] = {(void*)&geom, (void*)&pairs, (void*)&ctrl, (void*)&fp, (void*)&jkr_delta, (void*)&jkr_radius,
                    (void*)&jbuf, (void*)&surv, (void*)&al, (void*)&spv, (void*)&mlp_w, (void*)&flow};
    const cudaError_t e = launch_shape(fn, shape, PS_T, args, st);
    if (with_sum)
        k_pair_sum_rows<<<max(cdiv(cap_cells, 128), 1), 128, 0, st>>>(al.row_ptr, al.n_act, ctrl, jbuf, fcc, f32);
    return e;
}

// the reference's 2-D dE/dq (cellCellRepulsiveForces + cellCellAdhesiveForces) from the
// pair sums F = sum p and S = sum s p: torque S - (n . S) n at the current orientation
__global__ void k_pair_dEdq_2d(const Geom* __restrict__ geom, const Gen6* __restrict__ fcc, const Ctrl* ctrl,
                               double* cm)
{
    const int n = ctrl->n;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    {
        const Geom g = load_geom(geom, i);
        const Gen6 f = fcc[i];
        const double w = g.nx * f.f[3] + g.ny * f.f[4];
        cm[i] = f.f[0];
        cm[(size_t)n + i] = f.f[1];
        cm[(size_t)2 * n + i] = f.f[3] - w * g.nx;
        cm[(size_t)3 * n + i] = f.f[4] - w * g.ny;
    }
}

void launch_pair_dEdq_2d(const Geom* geom, const Gen6* fcc, const Ctrl* ctrl, double* cm, int cap_cells,
                         cudaStream_t st)
{
    k_pair_dEdq_2d<<<max(cdiv(cap_cells, 256), 1), 256, 0, st>>>(geom, fcc, ctrl, cm);
}

// Frame snapshot, at the end of an iteration: when the accepted step marked a frame,
// every cell's records go to ring slot frames_taken % slots, and the last block
// records the frame's time, iteration, cell count and lineage length.  The loop
// keeps running; the host downloads the slots when it writes the frames.
__global__ void k_frame_snapshot(const Geom* __restrict__ geom, const Vel* __restrict__ vel,
                                 const Phys* __restrict__ phys, Ctrl* ctrl, Geom* snap_geom, Vel* snap_vel,
                                 Phys* snap_phys, FrameInfo* info, int slots, int cap_cells,
                                 const double* __restrict__ feta, double* snap_feta)
{
    __shared__ bool last;
    // frame_due changes only in the last block below, after every block has passed here
    if (!ctrl->frame_due) return;
    const int n = ctrl->n;
    const size_t off = (size_t)(ctrl->frames_taken % slots) * cap_cells;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    {
        snap_geom[off + i] = geom[i];
        snap_vel[off + i] = vel[i];
        snap_phys[off + i] = phys[i];
        if (feta) snap_feta[off + i] = feta[i];
    }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        __threadfence();
        last = atomicAdd(&ctrl->frame_blocks, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (last && threadIdx.x == 0)
    {
        FrameInfo f;
        f.t = ctrl->t;
        f.iter = ctrl->iter;
        f.n = n;
        f.n_parents = ctrl->n_parents;
        f.pad = 0;
        info[ctrl->frames_taken % slots] = f;
        ctrl->frames_taken += 1;
        ctrl->frame_due = 0;
        ctrl->frame_blocks = 0u;
    }
}

void launch_frame_snapshot(const Geom* geom, const Vel* vel, const Phys* phys, Ctrl* ctrl, Geom* snap_geom,
                           Vel* snap_vel, Phys* snap_phys, FrameInfo* info, int slots, int cap_cells,
                           cudaStream_t st, const double* feta, double* snap_feta)
{
    const int blocks = max(min(cdiv(cap_cells, 256), 4 * 148), 1);
    k_frame_snapshot<<<blocks, 256, 0, st>>>(geom, vel, phys, ctrl, snap_geom, snap_vel, snap_phys, info, slots,
                                             cap_cells, feta, snap_feta);
}

__device__ __forceinline__ void loop_begin(Ctrl* c, int divides, int todo)
{
    c->todo = todo;
    c->hold = divides ? HOLD_START : HOLD_NONE;
    c->div_any = 0;
    c->rounds = 2 * todo + 4;
}
__global__ void k_loop_begin(Ctrl* c, int divides, int todo) { loop_begin(c, divides, todo); }
__global__ void k_loop_begin_all(Ctrl* const* ctrls, const int* divides, int n, int todo)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) loop_begin(ctrls[k], divides[k], todo);
}
__global__ void k_loop_round(Ctrl* c, unsigned long long cond_slow, unsigned long long cond_loop)
{
    const bool slow = c->hold != HOLD_NONE && c->todo > 0 && !c->halted;
    const int left = c->todo - (c->hold == HOLD_RETRY ? 1 : 0);
    c->rounds -= 1;
    cudaGraphSetConditional((cudaGraphConditionalHandle)cond_slow, slow ? 1u : 0u);
    cudaGraphSetConditional((cudaGraphConditionalHandle)cond_loop, left > 0 && !c->halted && c->rounds > 0 ? 1u : 0u);
}

void launch_loop_begin(Ctrl* ctrl, int divides, int todo, cudaStream_t st)
{
    k_loop_begin<<<1, 1, 0, st>>>(ctrl, divides, todo);
}
void launch_loop_begin_all(Ctrl* const* ctrls, const int* divides, int n, int todo, cudaStream_t st)
{
    k_loop_begin_all<<<cdiv(n, 128), 128, 0, st>>>(ctrls, divides, n, todo);
}
__global__ void k_retry_begin(const Ctrl* c, unsigned long long cond)
{
    cudaGraphSetConditional((cudaGraphConditionalHandle)cond, !loop_idle(c, FLOW_SLOW) && c->mode == MODE_RETRY ? 1u : 0u);
}
void launch_retry_begin(Ctrl* ctrl, unsigned long long cond, cudaStream_t st)
{
    k_retry_begin<<<1, 1, 0, st>>>(ctrl, cond);
}
void launch_loop_round(Ctrl* ctrl, unsigned long long cond_slow, unsigned long long cond_loop, cudaStream_t st)
{
    k_loop_round<<<1, 1, 0, st>>>(ctrl, cond_slow, cond_loop);
}

int attempt_blocks(int cap_cells) { return max(cdiv(cap_cells, AT_T), 1); }

void launch_attempt(int kind, const AttemptArgs& a, int dims, cudaStream_t st)
{
    switch (a.sp->s)
    {
        case 2: launch_attempt_2(kind, a, dims, st); break;
        case 4: launch_attempt_4(kind, a, dims, st); break;
        case 6: launch_attempt_6(kind, a, dims, st); break;
        case 7: launch_attempt_7(kind, a, dims, st); break;
        default: break;
    }
}

void launch_friction_rounds(int kind, const AttemptArgs& a, const int4* act, const int* fr_list, int* fmask, double R,
                            cudaStream_t st)
{
    switch (a.sp->s)
    {
        case 2: launch_friction_rounds_2(kind, a, act, fr_list, fmask, R, st); break;
        case 4: launch_friction_rounds_4(kind, a, act, fr_list, fmask, R, st); break;
        case 6: launch_friction_rounds_6(kind, a, act, fr_list, fmask, R, st); break;
        case 7: launch_friction_rounds_7(kind, a, act, fr_list, fmask, R, st); break;
        default: break;
    }
}

__global__ void k_velocities_2d(const Geom* __restrict__ geom, const Phys* __restrict__ phys,
                                const Gen6* __restrict__ fcc, const Ctrl* ctrl, StepParams sp, Gen6* v_out)
{
    const int n = ctrl->n;
    const double nz[4] = {0.0, 0.0, 0.0, 0.0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    {
        const Geom g = load_geom(geom, i);
        const double y[6] = {g.rx, g.ry, g.rz, g.nx, g.ny, g.nz};
        const Phys ph = phys[i];
        Gen6 out;
        velocity_2d(y, cell_drag_2d(sp, ph.l, ph.eta0, ph.eta1), load_gen6(fcc, i), nz, out.f);
        v_out[i] = out;
    }
}

__global__ void k_velocities(const Geom* __restrict__ geom, const Vel* __restrict__ vel,
                             const Phys* __restrict__ phys, const Gen6* __restrict__ fcc, const Ctrl* ctrl,
                             StepParams sp, Gen6* v_out)
{
    const int n = ctrl->n;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    {
        const Geom g = load_geom(geom, i);
        const double y[6] = {g.rx, g.ry, g.rz, g.nx, g.ny, g.nz};
        const bool a2 = y[5] < sp.mp.nz_threshold;
        double f0[6];
        base_force<false>(sp, load_gen6(fcc, i), 0, 0, i, f0);
        Gen6 out;
        const Phys ph = phys[i];
        CellDrag d = cell_drag(ph.l, ph.eta0);
        if (sp.mixed)
            cell_velocity<true>(sp.mp, a2, y, ph.l, g.h, ph.eta0, ph.eta1, ph.sigma0, d, vel + i, f0, out.f);
        else
            cell_velocity<false>(sp.mp, a2, y, ph.l, g.h, ph.eta0, ph.eta1, ph.sigma0, d, vel + i, f0, out.f);
        v_out[i] = out;
    }
}

void launch_velocities(const Geom* geom, const Vel* vel, const Phys* phys, const Gen6* fcc,
                       const Ctrl* ctrl, const StepParams& sp, Gen6* v_out, int cap_cells,
                       cudaStream_t st, int dims)
{
    if (dims == 2)
    {
        k_velocities_2d<<<max(cdiv(cap_cells, 128), 1), 128, 0, st>>>(geom, phys, fcc, ctrl, sp, v_out);
        return;
    }
    k_velocities<<<max(cdiv(cap_cells, 128), 1), 128, 0, st>>>(geom, vel, phys, fcc, ctrl, sp, v_out);
}

// growCells (growth.hpp:51-57)
__global__ void k_grow(Geom* geom, Phys* phys, const Ctrl* ctrl, double R, double dt)
{
    const int n = ctrl->n;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    {
        double l = phys[i].l;
        l += phys[i].growth * (4 * R / 3 + l) * dt;
        phys[i].l = l;
        geom[i].h = l / 2;
    }
}

void launch_grow(Geom* geom, Phys* phys, const Ctrl* ctrl, double R, double dt, int cap_cells,
                 cudaStream_t st)
{
    k_grow<<<max(cdiv(cap_cells, 256), 1), 256, 0, st>>>(geom, phys, ctrl, R, dt);
}

// ---------------------------------------------------------------------------
// Neighbor table in the reference's row order (i ascending, j < i ascending)
// ---------------------------------------------------------------------------
__global__ void k_count_lower(const Ctrl* ctrl, const int* row_ptr, const int* col, int* cnt)
{
    const int n = ctrl->n;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    {
        int c = 0;
        for (int k = row_ptr[i]; k < row_ptr[i + 1]; ++k) c += col[k] < i;
        cnt[i] = c;
    }
}

void launch_count_lower(const Ctrl* ctrl, const int* row_ptr, const int* col, int* cnt,
                        int cap_cells, cudaStream_t st)
{
    k_count_lower<<<max(cdiv(cap_cells, 256), 1), 256, 0, st>>>(ctrl, row_ptr, col, cnt);
}

// 3-D rows (i, j, dx, dy, dz, si, sj); 2-D rows (i, j, dx, dy, si, sj)
__global__ void k_table_rows(const Ctrl* ctrl, const int* row_ptr, const int* col, const int* pos,
                             const Geom* __restrict__ geom, double* out, int ld, int dims)
{
    const int n = ctrl->n;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    {
        int p = pos[i];
        Geom gi = load_geom(geom, i);
        for (int k = row_ptr[i]; k < row_ptr[i + 1]; ++k)
        {
            int j = col[k];
            if (j >= i) continue;
            Dist d = dist_geom(gi, load_geom(geom, j));
            out[p] = i; out[(size_t)ld + p] = j;
            out[(size_t)2 * ld + p] = d.dx; out[(size_t)3 * ld + p] = d.dy;
            if (dims == 2)
            {
                out[(size_t)4 * ld + p] = d.s; out[(size_t)5 * ld + p] = d.t;
            }
            else
            {
                out[(size_t)4 * ld + p] = d.dz;
                out[(size_t)5 * ld + p] = d.s; out[(size_t)6 * ld + p] = d.t;
            }
            ++p;
        }
    }
}

void launch_table_rows(const Ctrl* ctrl, const int* row_ptr, const int* col, const int* pos,
                       const Geom* geom, double* out, int ld, int cap_cells, cudaStream_t st, int dims)
{
    k_table_rows<<<max(cdiv(cap_cells, 128), 1), 128, 0, st>>>(ctrl, row_ptr, col, pos, geom, out, ld, dims);
}

}   // namespace abm
