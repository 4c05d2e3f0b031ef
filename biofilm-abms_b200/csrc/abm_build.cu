// Neighbor set and division on the device, one cooperative launch.
//
// Neighbor set (getCellNeighbors, mechanics.hpp:520-593), in phases with a barrier over the
// launch's blocks between them:
//   bounding box -> grid -> counting sort of the cells by bin
//   pair search -> row offsets and the attempt order -> CSR rows sorted by neighbor index
//   -> pair records (i, j < i, entry of j in row i, entry of i in row j) in bin order
// Division (abm_divide.cuh) before it, when cells exceed the division length.
//
// The rebuild was 21 kernels, the division another 12, a few microseconds of launch, ramp and
// tail each against little work (a growing colony divides, and so rebuilds, every few
// iterations).  A grid barrier costs 1.6 us up to 8 blocks and 2.7 us at 296, a cluster's
// hardware barrier 0.4 us, so colonies of up to BUILD_CLUSTER_CELLS cells run as one cluster
// of 16 blocks, which also needs no cooperative launch (those wait for the whole chip when
// the colonies of a batch share it).
#include "abm_grid.cuh"
#include "abm_divide.cuh"
#include <climits>

namespace abm {

const int BD_T = 512;                       // threads per block
const int BD_WARPS = BD_T / 32;
const int BD_SEARCH = 8;                    // lanes per cell in the pair search
const int BD_ROW = 8;                       // lanes per row of the CSR passes
const int SEARCH_ROWS = 16;                 // rows of bins taken at a time (a cell has 13)
const int SEARCH_AHEAD = 4;                 // candidates a lane loads at once
const int SEARCH_QUEUE = 32 + 32 * SEARCH_AHEAD;
const int FLAG_BIT = 1 << 30;               // attempt-order class beside a cell's entry count

// A bounding box in FP32, rounded outwards: the smallest and largest centre coordinates,
// the largest half-length and reach, as integers in the order of the floats so that a warp
// reduces each with one instruction (the doubles took 80 shuffles).
struct Box { int lo[3], hi[3], h, reach; };

struct BuildShared {
    Box box[BD_WARPS];
    int warp_sum[BD_WARPS], warp_flag[BD_WARPS];
    // pair search: candidate positions of each warp; each cell's rows of bins, as the first
    // position of a row and the candidates before it
    int q_a[BD_WARPS][SEARCH_QUEUE], q_b[BD_WARPS][SEARCH_QUEUE];
    int row_at[BD_T / BD_SEARCH][SEARCH_ROWS], row_before[BD_T / BD_SEARCH][SEARCH_ROWS + 1];
    Grid grid;
};

// ---------------------------------------------------------------------------
// Block reductions and scans
// ---------------------------------------------------------------------------
__device__ __forceinline__ int ord_int(float x) { const int b = __float_as_int(x); return b >= 0 ? b : b ^ 0x7fffffff; }
__device__ __forceinline__ float int_ord(int b) { return __int_as_float(b >= 0 ? b : b ^ 0x7fffffff); }

__device__ __forceinline__ Box empty_box()
{
    Box b;
    for (int k = 0; k < 3; ++k) { b.lo[k] = INT_MAX; b.hi[k] = INT_MIN; }
    b.h = b.reach = 0;
    return b;
}
// NaN coordinates are left out
__device__ __forceinline__ void box_of(Box& b, const Geom& g)
{
    const double r[3] = {g.rx, g.ry, g.rz};
    for (int k = 0; k < 3; ++k)
        if (!isnan(r[k]))
        {
            b.lo[k] = min(b.lo[k], ord_int(__double2float_rd(r[k])));
            b.hi[k] = max(b.hi[k], ord_int(__double2float_ru(r[k])));
        }
    b.h = max(b.h, ord_int(__double2float_ru(fmax(g.h, 0.0))));
    b.reach = max(b.reach, ord_int(fmaxf(segment_reach(g.h, g.nx, g.ny, g.nz), 0.f)));
}
__device__ __forceinline__ Box join(Box b, const Box& o)
{
    for (int k = 0; k < 3; ++k) { b.lo[k] = min(b.lo[k], o.lo[k]); b.hi[k] = max(b.hi[k], o.hi[k]); }
    b.h = max(b.h, o.h);
    b.reach = max(b.reach, o.reach);
    return b;
}
__device__ __forceinline__ Box warp_join(Box b)
{
    const unsigned full = 0xffffffffu;
    for (int k = 0; k < 3; ++k) { b.lo[k] = __reduce_min_sync(full, b.lo[k]); b.hi[k] = __reduce_max_sync(full, b.hi[k]); }
    b.h = __reduce_max_sync(full, b.h);
    b.reach = __reduce_max_sync(full, b.reach);
    return b;
}
// over the block, in every thread
__device__ __forceinline__ Box block_join(Box b, BuildShared& sh)
{
    b = warp_join(b);
    if ((threadIdx.x & 31) == 0) sh.box[threadIdx.x >> 5] = b;
    __syncthreads();
    b = warp_join((threadIdx.x & 31) < BD_WARPS ? sh.box[threadIdx.x & 31] : empty_box());
    __syncthreads();
    return b;
}

// exclusive prefix of (a, b) over the block, and the totals
__device__ __forceinline__ int2 block_scan(int2 v, BuildShared& sh, int2& total)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int2 x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const int a = __shfl_up_sync(0xffffffffu, x.x, o), b = __shfl_up_sync(0xffffffffu, x.y, o);
        if (lane >= o) { x.x += a; x.y += b; }
    }
    if (lane == 31) { sh.warp_sum[wid] = x.x; sh.warp_flag[wid] = x.y; }
    __syncthreads();
    int2 off = make_int2(0, 0);
    total = make_int2(0, 0);
#pragma unroll
    for (int w = 0; w < BD_WARPS; ++w)
    {
        if (w < wid) { off.x += sh.warp_sum[w]; off.y += sh.warp_flag[w]; }
        total.x += sh.warp_sum[w]; total.y += sh.warp_flag[w];
    }
    __syncthreads();
    return make_int2(off.x + x.x - v.x, off.y + x.y - v.y);
}

// Sum of part[0 .. blockIdx.x) and of all of them: where this block's chunk starts
__device__ __forceinline__ void chunk_offset(const int2* part, int nb, BuildShared& sh, int2& before, int2& all)
{
    int2 lo = make_int2(0, 0), t = lo;
    for (int b = threadIdx.x; b < nb; b += BD_T)
    {
        const int2 p = part[b];
        t.x += p.x; t.y += p.y;
        if (b < (int)blockIdx.x) { lo.x += p.x; lo.y += p.y; }
    }
    int2 total;
    block_scan(lo, sh, total);
    before = total;
    block_scan(t, sh, total);
    all = total;
}

// ---------------------------------------------------------------------------
// Cell list
// ---------------------------------------------------------------------------
__device__ __forceinline__ int bin_coord(double x, double x0, double inv_edge, int nb)
{
    int b = (int)floor((x - x0) * inv_edge);
    return b < 0 ? 0 : (b >= nb ? nb - 1 : b);
}

// The grid from the bounding box: bins of half the largest distance a pair can have (plus a
// part in 1e6 for the rounding of the bin coordinates), so that a cell looks two bins around;
// larger where the box would need more than cap_bins.  A box that no grid of cap_bins bins
// can hold is an overflow.
__device__ __forceinline__ Grid make_grid(const Box& b, const BuildArgs& a, bool& bad)
{
    double lo[3], hi[3];
    const double maxh = int_ord(b.h), reach = int_ord(b.reach);
    for (int k = 0; k < 3; ++k)
    {
        lo[k] = b.lo[k] == INT_MAX ? 0.0 : (double)int_ord(b.lo[k]);
        hi[k] = b.hi[k] == INT_MIN ? 0.0 : (double)int_ord(b.hi[k]);
    }
    // an axis without any number spans [0, 0], and an infinite extent, or one no grid of
    // cap_bins bins can hold, is an overflow
    bad = false;
    for (int k = 0; k < 3; ++k)
    {
        if (!(lo[k] <= hi[k])) { lo[k] = 0; hi[k] = 0; }
        if (!(hi[k] - lo[k] < 1e290)) bad = true;
    }
    Grid g;
    // the pair test is |r_j - r_i| < prefilter and |d| < threshold, |d| >= |r_j - r_i| less
    // both reaches
    // (a prefilter that no pair passes still needs bins of some size)
    g.reach = fmax(fmin(a.bp.prefilter, a.bp.threshold + 2 * reach + 1e-3), 1e-3);
    double e = 0.5 * g.reach * (1 + 1e-6);
    double nb[3] = {1.0, 1.0, 1.0};
    for (int tries = 0; tries < 68 && !bad; ++tries)
    {
        for (int k = 0; k < 3; ++k) nb[k] = floor((hi[k] - lo[k]) / e) + 1;
        if (nb[0] * nb[1] * nb[2] <= (double)a.cap_bins) break;
        e *= 1.5;
    }
    if (bad || !(nb[0] * nb[1] * nb[2] <= (double)a.cap_bins))
    {
        bad = true;
        for (int k = 0; k < 3; ++k) { nb[k] = 1.0; lo[k] = 0.0; hi[k] = 0.0; }
    }
    g.x0 = lo[0]; g.y0 = lo[1]; g.z0 = lo[2]; g.edge = e; g.inv_edge = 1.0 / e;
    g.nx = (int)nb[0]; g.ny = (int)nb[1]; g.nz = (int)nb[2];
    g.nbins = g.nx * g.ny * g.nz;
    g.max_half_l = maxh;
    g.max_reach = (float)reach;
    // FP32 coordinates from the box's corner: a difference of two errs by less than
    // 2 sqrt(3) 2^-24 of the extent, and the clipping of a row by a few times that
    const double ext = fmax(fmax(hi[0] - lo[0], hi[1] - lo[1]), hi[2] - lo[2]);
    g.margin = (float)(1e-4 + ext * (1.0 / 1048576));
    return g;
}

__device__ __forceinline__ bool build_barrier(const BuildArgs& a, int nb)
{
    if (a.cluster)
    {
        cluster_barrier();
        return true;
    }
    return grid_barrier(a.bar, nb, a.ctrl);
}

// this block's part of the bounding box
__device__ __forceinline__ void put_box(const BuildArgs& a, const Box& b, BuildShared& sh)
{
    const Box all = block_join(b, sh);
    if (threadIdx.x == 0) reinterpret_cast<Box*>(a.bbox)[blockIdx.x] = all;
}

// Sort the n cells by bin, from the blocks' bounding boxes (behind a barrier): bin_start
// (nx + 1 entries per row of bins along x), sorted_cell, sorted_pos (FP32 position from the
// box's corner and reach), key.  The bins of a row are contiguous, in order; the rows lie in
// any order, taken from one counter, so that no scan over all bins is needed.  bin_count is
// zero on entry and on return.  Barriers: 3, the last at the end.  False: a wait ran out.
__device__ bool cell_list(const BuildArgs& a, int n, int nb, BuildShared& sh, bool& bad)
{
    const int gt = blockIdx.x * BD_T + threadIdx.x, gs = nb * BD_T;
    Box box = empty_box();
    for (int b = threadIdx.x; b < nb; b += BD_T) box = join(box, reinterpret_cast<const Box*>(a.bbox)[b]);
    const Grid g = make_grid(block_join(box, sh), a, bad);
    if (threadIdx.x == 0)
    {
        sh.grid = g;
        if (blockIdx.x == 0)
        {
            if (bad) atomicOr(&a.ctrl->status, (int)ST_BIN_OVERFLOW);
            a.ctrl->n_pairs = 0;
            a.ctrl->n_sorted = 0;
            a.ctrl->no_table = bad;
        }
    }
    for (int i = gt; i < n; i += gs)
    {
        const Geom c = a.geom[i];
        const int bx = bin_coord(c.rx, g.x0, g.inv_edge, g.nx);
        const int by = bin_coord(c.ry, g.y0, g.inv_edge, g.ny);
        const int bz = bin_coord(c.rz, g.z0, g.inv_edge, g.nz);
        const int k = (bz * g.ny + by) * g.nx + bx;
        a.key[i] = k;
        a.slot[i] = atomicAdd(&a.bin_count[k], 1);
        a.count[i] = 0;
    }
    if (!build_barrier(a, nb)) return false;
    // a warp per row of bins
    const int lane = threadIdx.x & 31, rows = g.ny * g.nz;
    for (int r = gt >> 5; r < rows; r += gs >> 5)
    {
        int total = 0;
        for (int x = lane; x < g.nx; x += 32) total += a.bin_count[r * g.nx + x];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
        int at = 0;
        if (lane == 0 && total) at = atomicAdd(&a.ctrl->n_sorted, total);
        at = __shfl_sync(0xffffffffu, at, 0);
        for (int x0 = 0; x0 < g.nx; x0 += 32)
        {
            const int x = x0 + lane;
            const int m = x < g.nx ? a.bin_count[r * g.nx + x] : 0;
            int s = m;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
            {
                const int y = __shfl_up_sync(0xffffffffu, s, o);
                if (lane >= o) s += y;
            }
            if (x < g.nx)
            {
                a.bin_start[r * (g.nx + 1) + x] = at + s - m;
                a.bin_count[r * g.nx + x] = 0;
            }
            at += __shfl_sync(0xffffffffu, s, 31);
        }
        if (lane == 0) a.bin_start[r * (g.nx + 1) + g.nx] = at;
    }
    if (!build_barrier(a, nb)) return false;
    for (int i = gt; i < n; i += gs)
    {
        const int k = a.key[i];
        const int pos = a.bin_start[k + k / g.nx] + a.slot[i];
        const Geom c = a.geom[i];
        a.sorted_cell[pos] = i;
        a.sorted_key[pos] = k;
        a.sorted_dir[pos] = make_float4((float)c.nx, (float)c.ny, (float)c.nz, (float)c.h);
        a.sorted_pos[pos] = make_float4((float)(c.rx - g.x0), (float)(c.ry - g.y0), (float)(c.rz - g.z0),
                                        segment_reach(c.h, c.nx, c.ny, c.nz));
    }
    return build_barrier(a, nb);
}

// ---------------------------------------------------------------------------
// Pair search.  BD_SEARCH lanes per cell walk the bins around it, half of them, so that each
// unordered pair is met once: the rest of its own row of bins and the rows after it, each
// clipped to the circle the cell can reach.  The lanes look up a cell's rows side by side and
// then walk them as one list, four loads each in flight: row after row, with its two bin
// offsets and its loads one behind the other, took 57 us at 20,000 cells.  A candidate is dropped only when, in FP32
// with the grid's margin, |r2 - r1| > threshold + both reaches, i.e. when its |d| is
// certainly >= threshold (segment_reach), or when the separating-axis bound says so (near_f;
// without it 28 candidates a cell went on to the exact test, for 7.5 neighbors, and that
// test took most of the time).  The survivors go to a queue of the warp and are
// evaluated 32 at a time, so that the exact FP64 distance runs on full warps.  A survivor is
// kept when it passes the reference's two tests: centre distance < threshold + Ldiv + 2R
// and segment distance < threshold (mechanics.hpp:548-577), evaluated with the larger index
// as cell 1, as the reference's j < i loop does.  Both cells' rows get the entry, in any
// order; the rows are sorted next.
//
// What bounds it: the FP32 sweep and its loads.  Bins of the whole reach and both directions of every pair
// took 264 us at 100,000 cells (372 candidates a cell, 96 us at 20,000 with one block per bin).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void add_entry(const BuildArgs& a, int i, int j)
{
    const int s = atomicAdd(&a.count[i], 1);
    if (s < a.bp.cap_per_cell) a.scratch[(size_t)i * a.bp.cap_per_cell + s] = j;
}

__device__ __forceinline__ void exact_pair(const BuildArgs& a, int p, int q)
{
    const int c1 = a.sorted_cell[p], c2 = a.sorted_cell[q];
    const int i = max(c1, c2), j = min(c1, c2);
    const Geom gi = a.geom[i], gj = a.geom[j];
    const double cd = xnorm(xsub(x3(gi.rx, gi.ry, gi.rz), x3(gj.rx, gj.ry, gj.rz)));
    if (!(cd < a.bp.prefilter)) return;
    const Dist d = dist_geom(gi, gj);
    if (xnorm(x3(d.dx, d.dy, d.dz)) < a.bp.threshold)
    {
        add_entry(a, i, j);
        add_entry(a, j, i);
    }
}

// A cell's row `r` of the half neighborhood: its own row first, then the rows after it
__device__ __forceinline__ void half_row(int r, int rings, int& dy, int& dz)
{
    const int w = 2 * rings + 1, q = r + rings;      // row (dy, dz) has q = dz w + dy + rings
    dz = q / w;
    dy = q % w - rings;
}

__device__ __forceinline__ void pair_search(const BuildArgs& a, int n, int nb, BuildShared& sh)
{
    const Grid& g = sh.grid;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const int per_warp = 32 / BD_SEARCH, sub = lane & (BD_SEARCH - 1), group = threadIdx.x / BD_SEARCH;
    const float thr = (float)a.bp.threshold + g.margin;
    const float edge = (float)g.edge, inv = (float)g.inv_edge;
    const int rings = max((int)ceil(g.reach * g.inv_edge), 1);
    const int n_rows = rings * (2 * rings + 1) + rings + 1;
    int* at = sh.row_at[group];
    int* before = sh.row_before[group];
    int qn = 0;                                     // this warp's queue length (warp-uniform)
    for (int base = (blockIdx.x * BD_WARPS + warp) * per_warp; base < n; base += nb * BD_WARPS * per_warp)
    {
        const int p = base + lane / BD_SEARCH;
        const bool valid = p < n;
        float4 c = make_float4(0.f, 0.f, 0.f, 0.f), dir = c;
        int bx = 0, by = 0, bz = 0;
        if (valid)
        {
            c = a.sorted_pos[p];
            dir = a.sorted_dir[p];
            const int k = a.sorted_key[p];
            bx = k % g.nx; by = (k / g.nx) % g.ny; bz = k / (g.nx * g.ny);
        }
        const float own = thr + c.w;
        const float far = own + g.max_reach + 1e-3f;     // no pair lies beyond
        for (int r0 = 0; r0 < n_rows; r0 += SEARCH_ROWS)
        {
            // the group's lanes look the rows up side by side
            __syncwarp();
            int carry = 0;
#pragma unroll
            for (int h = 0; h < SEARCH_ROWS; h += BD_SEARCH)
            {
                const int r = r0 + h + sub;
                int q = 0, len = 0;
                if (valid && r < n_rows)
                {
                    int dy, dz;
                    half_row(r, rings, dy, dz);
                    const int zz = bz + dz, yy = by + dy;
                    if (zz < g.nz && yy >= 0 && yy < g.ny)
                    {
                        // distance to the row of bins, then the part of it within reach
                        const float gz = dz ? fmaxf(zz * edge - c.z, 0.f) : 0.f;
                        const float gy = dy > 0 ? fmaxf(yy * edge - c.y, 0.f)
                                                : dy < 0 ? fmaxf(c.y - (yy + 1) * edge, 0.f) : 0.f;
                        const float w2 = far * far - gz * gz - gy * gy;
                        if (!(w2 < 0.f))
                        {
                            const float w = sqrtf(w2);
                            const int x_lo = max(max((int)floorf((c.x - w) * inv - 1e-3f), bx - rings), 0);
                            const int x_hi = min(min((int)floorf((c.x + w) * inv + 1e-3f), bx + rings), g.nx - 1);
                            const int row = (zz * g.ny + yy) * (g.nx + 1);
                            if (x_lo <= x_hi)
                            {
                                q = r ? a.bin_start[row + x_lo] : p + 1;
                                len = max(a.bin_start[row + x_hi + 1] - q, 0);
                            }
                        }
                    }
                }
                int x = len;
#pragma unroll
                for (int o = 1; o < BD_SEARCH; o <<= 1)
                {
                    const int y = __shfl_up_sync(0xffffffffu, x, o, BD_SEARCH);
                    if (sub >= o) x += y;
                }
                at[h + sub] = q;
                before[h + sub] = carry + x - len;
                carry += __shfl_sync(0xffffffffu, x, BD_SEARCH - 1, BD_SEARCH);
            }
            if (sub == 0) before[SEARCH_ROWS] = carry;
            __syncwarp();
            // then walk the candidates of all rows as one list
            int row = 0;
            for (int e0 = sub; __any_sync(0xffffffffu, e0 < carry); e0 += BD_SEARCH * SEARCH_AHEAD)
            {
                int q[SEARCH_AHEAD];
                float4 o[SEARCH_AHEAD];
#pragma unroll
                for (int u = 0; u < SEARCH_AHEAD; ++u)
                {
                    const int e = e0 + u * BD_SEARCH;
                    q[u] = -1;
                    if (e < carry)
                    {
                        while (e >= before[row + 1]) ++row;
                        q[u] = at[row] + (e - before[row]);
                        o[u] = a.sorted_pos[q[u]];
                    }
                }
#pragma unroll
                for (int u = 0; u < SEARCH_AHEAD; ++u)
                {
                    bool pass = false;
                    if (q[u] >= 0)
                    {
                        const float fx = o[u].x - c.x, fy = o[u].y - c.y, fz = o[u].z - c.z, L = own + o[u].w;
                        pass = !(fx * fx + fy * fy + fz * fz > L * L);
                        if (pass)
                            pass = near_f(dir, a.sorted_dir[q[u]], fx, fy, fz, thr + 1e-3f + 1e-5f * L);
                    }
                    const unsigned m = __ballot_sync(0xffffffffu, pass);
                    if (pass)
                    {
                        const int s = qn + __popc(m & lt);
                        sh.q_a[warp][s] = p;
                        sh.q_b[warp][s] = q[u];
                    }
                    qn += __popc(m);
                }
                while (qn >= 32)
                {
                    qn -= 32;
                    __syncwarp();
                    const int ea = sh.q_a[warp][qn + lane], eb = sh.q_b[warp][qn + lane];
                    __syncwarp();
                    exact_pair(a, ea, eb);
                }
            }
        }
    }
    __syncwarp();
    if (lane < qn) exact_pair(a, sh.q_a[warp][lane], sh.q_b[warp][lane]);
}

// ---------------------------------------------------------------------------
// CSR and the pair records
// ---------------------------------------------------------------------------
// Attempt order (3-D): the cells whose velocity takes the full surface solve (area integrals,
// mechanics.hpp:2254-2309) first, then the others, each group in index order, so that the
// warps of an attempt mostly run one of the three branches of getVelocities
// (mechanics.hpp:2011-2347) instead of all of them.  Made at every rebuild from the cells of
// that moment; a cell that changes branch before the next costs only divergence.  The order
// changes no per-cell result.
__device__ __forceinline__ bool full_solve(const Geom& g, const MechParams& P)
{
    const bool a2 = g.nz < P.nz_threshold;
    const bool contact = a2 ? (g.rz < P.R) : ((g.rz - g.h * g.nz < P.R) || (g.rz + g.h * g.nz < P.R));
    return !P.no_surface && !a2 && contact;
}

// sum over the BD_ROW lanes of a row's group
__device__ __forceinline__ int group_sum(int v)
{
#pragma unroll
    for (int o = BD_ROW / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// row_ptr, the attempt order and the rows themselves, a contiguous chunk of cells per block:
// the chunks' totals, then behind a barrier each block's offsets, then its rows, sorted
// ascending (the deterministic order of the force sums; the reference's table is i-major,
// j ascending): an entry's rank is the number of smaller entries of its row.  Barriers: 1
// between, 1 at the end.
// When a cell has more neighbors than a row holds, every row is left empty, as where no grid
// holds the cells: rows cut off one by one would hold entries without their partners' entries,
// and neither the number of pair records nor the slots of their shares would be right.
__device__ bool make_rows(const BuildArgs& a, int n, int nb, BuildShared& sh, bool bad, int& n_dir)
{
    const int chunk = (n + nb - 1) / nb;
    const int c0 = min((int)blockIdx.x * chunk, n), c1 = min(c0 + chunk, n);
    int2 total;
    {
        int2 s = make_int2(0, 0);
        bool over = false;
        for (int i = c0 + threadIdx.x; i < c1; i += BD_T)
        {
            int m = bad ? 0 : a.count[i];
            if (m > a.bp.cap_per_cell) { over = true; m = a.bp.cap_per_cell; }
            const int f = a.order && full_solve(a.geom[i], a.mp);
            a.count[i] = m | (f ? FLAG_BIT : 0);
            s.x += m; s.y += f;
        }
        if (over)
        {
            atomicOr(&a.ctrl->status, (int)ST_NBR_OVERFLOW);
            a.ctrl->no_table = 1;
        }
        block_scan(s, sh, total);
        if (threadIdx.x == 0) a.part[blockIdx.x] = total;
    }
    if (!build_barrier(a, nb)) return false;
    const int no_table = __ldcg(&a.ctrl->no_table);        // under way beside the offsets' loads
    int2 off, all;
    chunk_offset(a.part, nb, sh, off, all);
    if (no_table)
    {
        off.x = all.x = 0;
        for (int i = c0 + threadIdx.x; i < c1; i += BD_T) a.count[i] &= FLAG_BIT;
        __syncthreads();
    }
    for (int i0 = c0; i0 < c1; i0 += BD_T)
    {
        const int i = i0 + threadIdx.x;
        const int v = i < c1 ? a.count[i] : 0;
        const int2 mine = make_int2(v & ~FLAG_BIT, (v & FLAG_BIT) ? 1 : 0);
        const int2 ex = block_scan(mine, sh, total);
        if (i < c1)
        {
            a.row_ptr[i] = off.x + ex.x;
            // full solves first: all.y of them
            if (a.order) a.order[mine.y ? off.y + ex.y : all.y + (i - (off.y + ex.y))] = i;
        }
        off.x += total.x; off.y += total.y;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) a.row_ptr[n] = all.x;
    n_dir = all.x;
    __syncthreads();
    const int lane = threadIdx.x & (BD_ROW - 1), group = threadIdx.x / BD_ROW;
    for (int i0 = c0; i0 < c1; i0 += BD_T / BD_ROW)
    {
        const bool valid = i0 + group < c1;
        const int i = valid ? i0 + group : c0;
        const int r0 = a.row_ptr[i], len = valid ? a.count[i] & ~FLAG_BIT : 0;
        const int* src = a.scratch + (size_t)i * a.bp.cap_per_cell;
        // warp-uniform rounds, so that the shuffles cover all lanes
        int longest = len;
#pragma unroll
        for (int o = 16; o >= BD_ROW; o >>= 1) longest = max(longest, __shfl_xor_sync(0xffffffffu, longest, o));
        int low = 0;
        for (int e = 0; e < longest; e += BD_ROW)
        {
            const int v = e + lane < len ? src[e + lane] : INT_MAX;
            int rank = 0;
            for (int b = 0; b < longest; b += BD_ROW)
            {
                const int w = b + lane < len ? src[b + lane] : INT_MAX;
#pragma unroll
                for (int q = 0; q < BD_ROW; ++q) rank += __shfl_sync(0xffffffffu, w, q, BD_ROW) < v;
            }
            if (e + lane < len)
            {
                a.col[r0 + rank] = v;
                low += v < i;
            }
        }
        low = group_sum(low);
        if (valid && lane == 0) a.lower_end[i] = r0 + low;
    }
    return build_barrier(a, nb);
}

// rows that the caller gave: only where their lower part ends
__device__ __forceinline__ void lower_ends(const BuildArgs& a, int n, int nb)
{
    for (int i = blockIdx.x * BD_T + threadIdx.x; i < n; i += nb * BD_T)
    {
        int e = a.row_ptr[i];
        while (e < a.row_ptr[i + 1] && a.col[e] < i) ++e;
        a.lower_end[i] = e;
    }
}

// The pair records, cells in bin order (`sorted`) or index order: pairs of one region of
// space are screened together, so each cell's record is fetched once and reused from the
// caches by its neighbors' pairs.  The partner's entry by binary search in its row; 2-D
// adhesion: to_adhere (2D/include/simulation.hpp:242-258, one group in the adhesion map) of
// the (i, j) row, dist > R + Rcell and < 2R.
__device__ __forceinline__ void pair_records(const BuildArgs& a, int n, int nb, bool sorted)
{
    const int lane = threadIdx.x & 31, sub = lane & (BD_ROW - 1);
    const int rows = nb * BD_T / BD_ROW;
    for (int p0 = (blockIdx.x * BD_T + threadIdx.x) / BD_ROW; p0 - lane / BD_ROW < n; p0 += rows)
    {
        const bool valid = p0 < n;
        const int i = valid ? (sorted ? a.sorted_cell[p0] : p0) : 0;
        const int r0 = a.row_ptr[i], low = valid ? a.lower_end[i] - r0 : 0;
        // one slot request per warp: the group's offset among the warp's rows
        int off = 0, all = 0;
#pragma unroll
        for (int s = 0; s < 32; s += BD_ROW)
        {
            const int m = __shfl_sync(0xffffffffu, low, s);
            if (s < (lane & ~(BD_ROW - 1))) off += m;
            all += m;
        }
        int pos = 0;
        if (lane == 0 && all) pos = atomicAdd(&a.ctrl->n_pairs, all);
        pos = __shfl_sync(0xffffffffu, pos, 0) + off;
        for (int e = sub; e < low; e += BD_ROW)
        {
            const int j = a.col[r0 + e];
            int x = a.row_ptr[j], y = a.row_ptr[j + 1];
            while (x < y) { const int mid = (x + y) >> 1; if (a.col[mid] < i) x = mid + 1; else y = mid; }
            // a pair that the caller's rows list more than once: each of its entries with another
            // one of the partner's
            if (!sorted)
                for (int q = e; q > 0 && a.col[r0 + q - 1] == j; --q) ++x;
            a.pairs[pos + e] = make_int4(i, j, r0 + e, x);
            if (a.adhere)
            {
                const Dist d = dist_geom(a.geom[i], a.geom[j]);
                const double dist = xnorm(x3(d.dx, d.dy, d.dz));
                a.adhere[r0 + e] = (dist > a.mp.R + a.mp.Rcell && dist < 2 * a.mp.R) ? 1 : 0;
                a.adhere[x] = 0;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Division.  n grows by the mothers, whose number is `divided`; on return the blocks' bounding
// boxes are those of the new population.  Ends with a barrier.  False: a wait ran out.
// ---------------------------------------------------------------------------
__device__ bool divide_cells(const BuildArgs& a, int& n, int nb, BuildShared& sh, int& divided)
{
    Ctrl* ctrl = a.ctrl;
    divided = 0;
    // mothers in ascending index order (divideMaxLength, growth.hpp:66-71): a chunk per block
    const int chunk = (n + nb - 1) / nb;
    const int c0 = min((int)blockIdx.x * chunk, n), c1 = min(c0 + chunk, n);
    int2 total;
    {
        int2 s = make_int2(0, 0);
        Box v = empty_box();
        for (int i = c0 + threadIdx.x; i < c1; i += BD_T)
        {
            const int f = a.phys[i].l > a.dp.Ldiv;
            a.flags[i] = f;
            s.x += f;
            box_of(v, a.geom[i]);
        }
        block_scan(s, sh, total);
        if (threadIdx.x == 0) a.part[blockIdx.x] = total;
        put_box(a, v, sh);
    }
    if (!build_barrier(a, nb)) return false;
    if (blockIdx.x == 0 && threadIdx.x == 0)
    {
        // every block has read them
        atomicAnd(&ctrl->halted, ~(int)HALT_CELLS);
        ctrl->hold = HOLD_NONE;
        ctrl->n_divided = 0;
    }
    int2 off, all;
    chunk_offset(a.part, nb, sh, off, all);
    int nd = all.x;
    if (nd > 0 && n + nd > a.cap_cells)
    {
        if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(&ctrl->status, (int)ST_CELL_OVERFLOW);
        nd = 0;
    }
    if (nd == 0) return true;
    for (int i0 = c0; i0 < c1; i0 += BD_T)
    {
        const int i = i0 + threadIdx.x;
        const int f = i < c1 ? a.flags[i] : 0;
        const int2 ex = block_scan(make_int2(f, 0), sh, total);
        if (f) a.mothers[off.x + ex.x] = i;
        off.x += total.x;
    }
    bool bad;
    if (!cell_list(a, n, nb, sh, bad)) return false;
    const int iter = ctrl->iter, np = ctrl->n_parents;
    const double t = ctrl->t;
    int tries = 0;
    for (bool done = false; !done;)
    {
        div_draw_phase(a, sh.grid, nd, nb, iter, tries);
        if (!build_barrier(a, nb)) return false;
        div_near_phase(a, sh.grid, nd, nb);
        if (!build_barrier(a, nb)) return false;
        // satisfied mothers so far: every block counts them all
        int2 s = make_int2(0, 0);
        for (int k = threadIdx.x; k < nd; k += BD_T)
        {
            const int ok = a.sat[k] || (a.check[k] == 1 && a.ok[2 * k] && a.ok[2 * k + 1]);
            if (ok) a.sat[k] = 1;
            s.x += ok;
        }
        block_scan(s, sh, total);
        tries += 1;
        // while (ntries == 0 || (ntries < 10 && satisfied < n_divide))  (growth.hpp:252)
        done = total.x >= nd || tries >= DIV_TRIES;
    }
    // the new population's boxes from the cells that stay and the daughters, beside the commit
    Box v = empty_box();
    for (int i = c0 + threadIdx.x; i < c1; i += BD_T)
        if (!a.flags[i]) box_of(v, a.geom[i]);
    for (int k = blockIdx.x * BD_T + threadIdx.x; k < nd; k += nb * BD_T)
    {
        box_of(v, a.d1[k]);
        box_of(v, a.d2[k]);
    }
    put_box(a, v, sh);
    div_commit_phase(a, n, nd, nb, np, t, iter);
    if (!build_barrier(a, nb)) return false;
    if (blockIdx.x == 0 && threadIdx.x == 0)
    {
        ctrl->n = n + nd;
        ctrl->n_parents = np + 2 * nd;
        ctrl->divisions += nd;
        ctrl->div_events += 1;
        ctrl->last_div_tries = tries;
        ctrl->n_divided = nd;
        ctrl->screen_valid = ctrl->path_valid = 0;     // new cells: the active pair list is stale
    }
    n += nd;
    divided = nd;
    return true;
}

// ---------------------------------------------------------------------------
// The launch.  `what`: BUILD_NEIGHBORS rebuilds the neighbor set; BUILD_DIVIDE divides the
// cells longer than the division length; BUILD_GROWTH divides and, if any cell did, rebuilds;
// BUILD_RECORDS makes the pair records of a neighbor set that the caller gave (row_ptr, col).
// Inside the loop graph (flow not FLOW_STEP) BUILD_GROWTH leaves at once unless the last step
// asked for it (Ctrl::hold).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(BD_T, 1) k_build(const __grid_constant__ BuildArgs a, int what, int flow)
{
    __shared__ BuildShared sh;
    Ctrl* ctrl = a.ctrl;
    if (ctrl->halted & HALT_LOST) return;
    if (flow != FLOW_STEP && (ctrl->todo <= 0 || ctrl->hold != HOLD_START)) return;
    int n = ctrl->n;
    const int nb = gridDim.x;
    int n_dir = 0;
    bool bad = false;
    if (what == BUILD_RECORDS)
    {
        lower_ends(a, n, nb);
        if (blockIdx.x == 0 && threadIdx.x == 0) { ctrl->n_pairs = 0; ctrl->no_table = 0; }
        if (!build_barrier(a, nb)) return;
        pair_records(a, n, nb, false);
        if (blockIdx.x == 0 && threadIdx.x == 0) ctrl->screen_valid = ctrl->path_valid = 0;
        return;
    }
    if (what == BUILD_NEIGHBORS)
    {
        Box v = empty_box();
        for (int i = blockIdx.x * BD_T + threadIdx.x; i < n; i += nb * BD_T) box_of(v, a.geom[i]);
        put_box(a, v, sh);
        if (!build_barrier(a, nb)) return;
    }
    else
    {
        // terminate() at the top of the loop: no division and no step once n reaches the limit
        if (ctrl->halt_n > 0 && n >= ctrl->halt_n)
        {
            if (blockIdx.x == 0 && threadIdx.x == 0) { atomicOr(&ctrl->halted, (int)HALT_CELLS); ctrl->n_divided = 0; }
            return;
        }
        int divided;
        if (!divide_cells(a, n, nb, sh, divided)) return;
        if (what == BUILD_DIVIDE || divided == 0) return;
    }
    if (!cell_list(a, n, nb, sh, bad)) return;
    if (!bad) pair_search(a, n, nb, sh);
    if (!build_barrier(a, nb)) return;
    if (!make_rows(a, n, nb, sh, bad, n_dir)) return;
    pair_records(a, n, nb, true);
    if (blockIdx.x == 0 && threadIdx.x == 0)
    {
        ctrl->n_dir = n_dir;
        if (a.order) ctrl->n_order = n;
        ctrl->screen_valid = ctrl->path_valid = 0;     // a new pair list makes the active list stale
        ctrl->rebuilds += 1;
    }
}

// The blocks of a launch for about `cells` cells (more only take longer): one cluster of up to
// 16 for a small colony, else a cooperative grid of up to two per SM, BD_SEARCH threads a cell.
LaunchShape build_shape(int cells, int num_sms, int share)
{
    return make_shape((const void*)k_build, BD_T, (long long)cells * BD_SEARCH, cells <= BUILD_CLUSTER_CELLS, num_sms,
                      share);
}

cudaError_t launch_build(const BuildArgs& args, int what, const LaunchShape& shape, cudaStream_t st, int flow)
{
    BuildArgs a = args;
    a.cluster = shape.cluster;
    void* p[] = {(void*)&a, (void*)&what, (void*)&flow};
    return launch_shape((const void*)k_build, shape, BD_T, p, st);
}

}   // namespace abm
