// Cell-list build: cell hash, exclusive prefix sum, stable counting sort, SoA reorder.
//
// Reference: ParticleSystem.update_grid_id / PrefixSumExecutor.run / counting_sort
// (eng/particle_system.py:228-257).  The reference sorts an 800-byte struct with an
// atomic_sub in a parallel loop, so its within-cell order is nondeterministic; the serial
// order of that loop is a stable counting sort by cell (ascending old index inside a
// cell).  This file produces exactly that order:
//   k_hash      cell index per particle (truncating cast, eng/particle_system.py:216-226),
//               atomic arrival rank inside the cell;
//   scan        exclusive prefix sum of the G + 1 counts (the extra bin collects
//               particles whose flattened index falls outside [0, G));
//   k_scatter   perm[cell_start + rank] = old index (unstable inside a cell);
//   k_cell_sort_big (tsg_cellsort.cuh) orders cells above kSortSmall by old index in scenes
//               above kSortAll particles;
//   k_reorder64 ranks the others' particles by old index (tsg_cellrank.cuh; stable result),
//               gathers every persistent field into the other buffer set, writes the f32
//               prefilter positions and the flow / boundary index lists.
// Compiled with -fmad=false: the f64 cell arithmetic must round exactly like the oracle's.
#include <cstdio>

#include "tsg_cellrank.cuh"
#include "tsg_cellsort.cuh"
#include "tsg_internal.h"
#include "tsg_pairs64.cuh"

namespace tsg {

namespace {

constexpr int TPB = 256;

__global__ void k_hash(Consts c, const double* __restrict__ x, int* __restrict__ cell_of,
                       int* __restrict__ rank, int* __restrict__ count, long long* __restrict__ cell0,
                       int* __restrict__ err) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    double xi[3];
    for (int d = 0; d < 3; ++d) xi[d] = x[(size_t)d * c.n + i];
    long long f = flat_cell(c, xi);
    cell0[i] = f;
    if (f < 0 || f >= c.G) {
        atomicOr(err, f != kNoCell ? TSG_ERR_CELL_OOB : (TSG_ERR_CELL_OOB | TSG_ERR_NONFINITE));
        f = c.G;
    }
    cell_of[i] = (int)f;
    rank[i] = atomicAdd(&count[f], 1);
}

// ---- three-phase exclusive scan (tile sums, scan of sums, tile rescan) ----
constexpr int SCAN_ITEMS = 8;
constexpr int SCAN_TILE = TPB * SCAN_ITEMS;

__device__ __forceinline__ int warp_incl_scan(int v) {
    const unsigned lane = threadIdx.x & 31u;
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= (unsigned)o) v += y;
    }
    return v;
}

// Block-wide exclusive scan of one value per thread; every thread receives the total.
__device__ __forceinline__ int block_excl_scan(int v, int& total) {
    __shared__ int warp_sums[TPB / 32];
    __shared__ int s_total;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int incl = warp_incl_scan(v);
    if (lane == 31) warp_sums[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        int w = lane < TPB / 32 ? warp_sums[lane] : 0;
        int wi = warp_incl_scan(w);
        if (lane < TPB / 32) warp_sums[lane] = wi - w;
        if (lane == TPB / 32 - 1) s_total = wi;
    }
    __syncthreads();
    int r = incl - v + warp_sums[wid];
    total = s_total;
    __syncthreads();
    return r;
}

__global__ void k_tile_sums(const int* __restrict__ in, int n, int* __restrict__ tile_sum) {
    __shared__ int red[TPB / 32];
    const int base = blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_ITEMS;
    int s = 0;
    for (int k = 0; k < SCAN_ITEMS; ++k) if (base + k < n) s += in[base + k];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        int w = threadIdx.x < TPB / 32 ? red[threadIdx.x] : 0;
        for (int o = 16; o > 0; o >>= 1) w += __shfl_down_sync(0xffffffffu, w, o);
        if (threadIdx.x == 0) tile_sum[blockIdx.x] = w;
    }
}

// One block scans all tile sums in place (exclusive), looping over chunks of TPB.
__global__ void k_scan_tiles(int* __restrict__ tile_sum, int ntiles) {
    int total = 0;
    int carry = 0;
    for (int b = 0; b < ntiles; b += TPB) {
        int i = b + threadIdx.x;
        int v = i < ntiles ? tile_sum[i] : 0;
        int e = block_excl_scan(v, total);
        if (i < ntiles) tile_sum[i] = e + carry;
        carry += total;
    }
}

__global__ void k_tile_rescan(const int* __restrict__ in, int n, const int* __restrict__ tile_sum,
                              int* __restrict__ out) {
    int total = 0;
    const int base = blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_ITEMS;
    int v[SCAN_ITEMS];
    int s = 0;
    for (int k = 0; k < SCAN_ITEMS; ++k) { v[k] = base + k < n ? in[base + k] : 0; s += v[k]; }
    int e = block_excl_scan(s, total) + tile_sum[blockIdx.x];
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        if (base + k < n) out[base + k] = e;
        e += v[k];
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == blockDim.x - 1) out[n] = e;  // grand total
}

// One block scans up to SCAN_ONE counts (a 2D scene's grid): one launch instead of three whose
// few blocks each take a launch's latency.
constexpr int SCAN_ONE_TPB = 1024, SCAN_ONE_ITEMS = 16, SCAN_ONE = SCAN_ONE_TPB * SCAN_ONE_ITEMS;
__device__ __forceinline__ void scan_one(const int* __restrict__ in, int n, int* out) {
    __shared__ int warp_sums[SCAN_ONE_TPB / 32];
    const int per = (n + SCAN_ONE_TPB - 1) / SCAN_ONE_TPB, base = threadIdx.x * per;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int v[SCAN_ONE_ITEMS], s = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ONE_ITEMS; ++k) {
        v[k] = k < per && base + k < n ? in[base + k] : 0;
        s += v[k];
    }
    const int incl = warp_incl_scan(s);
    if (lane == 31) warp_sums[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        const int w = warp_sums[lane];
        warp_sums[lane] = warp_incl_scan(w) - w;
    }
    __syncthreads();
    int e = warp_sums[wid] + incl - s;
#pragma unroll
    for (int k = 0; k < SCAN_ONE_ITEMS; ++k) {
        if (k < per && base + k < n) out[base + k] = e;
        e += v[k];
    }
    if (threadIdx.x == SCAN_ONE_TPB - 1) out[n] = e;  // grand total
}
__global__ void __launch_bounds__(SCAN_ONE_TPB) k_scan_one(const int* __restrict__ in, int n, int* out) {
    scan_one(in, n, out);
}

// The same block goes on to place the particles of the smallest scenes (whose cells the reorder
// pass ranks whatever their size): one launch instead of two on the step's chain.  3,274
// particles, rollout of 40 steps with gradient: 9,993 -> 9,659 us; 9,144 particles, ten steps:
// 867 -> 878, so the line lies between.
constexpr int SCATTER_ONE = 4096;
__global__ void __launch_bounds__(SCAN_ONE_TPB) k_scan_scatter(const int* __restrict__ count, int nbins, int* cell_start,
                                                              int n, const int* __restrict__ cell_of,
                                                              const int* __restrict__ rank, int* __restrict__ perm) {
    scan_one(count, nbins, cell_start);
    __syncthreads();
#pragma unroll 4
    for (int i = threadIdx.x; i < n; i += SCAN_ONE_TPB) perm[cell_start[cell_of[i]] + rank[i]] = i;
}

// Places the particles in arrival order inside their cells and lists the cells above `small`
// particles, which k_cell_sort_big orders; k_reorder64 ranks the particles of the others.
__global__ void k_scatter(int n, const int* __restrict__ cell_of, const int* __restrict__ rank,
                          const int* __restrict__ cell_start, int* __restrict__ perm, int small,
                          int* __restrict__ big, int* __restrict__ nbig) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int c = cell_of[i], r = rank[i], b = cell_start[c];
    perm[b + r] = i;
    if (r == 0 && cell_start[c + 1] - b > small) big[atomicAdd(nbig, 1)] = c;
}

__device__ __forceinline__ void append(int* list, int* counter, bool pred, int value) {
    unsigned mask = __ballot_sync(0xffffffffu, pred);
    if (!mask) return;
    const int lane = threadIdx.x & 31;
    int leader = __ffs(mask) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(counter, __popc(mask));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (pred) list[base + __popc(mask & ((1u << lane) - 1u))] = value;
}

// vt_src / vt_dst (3 planes each, may be null): v_tmp carried with its particle.  The
// mu(I) first loop reads the dummy particles' v_tmp of the previous step before the
// boundary loop rewrites it (eng/solver_sph_muI.py:67-109), and the reference's
// array-of-structs sort moves it with the particle.
template <bool SOIL>
__global__ void k_reorder64(Consts c, const int* __restrict__ perm, Persist64 a, Persist64 b,
                            float4* __restrict__ pos32, float4* __restrict__ pos32l,
                            const int* __restrict__ cell_of, const int* __restrict__ cell_start, int small,
                            const long long* __restrict__ cell_src, long long* __restrict__ cell0,
                            unsigned char* __restrict__ cell_flow, int* __restrict__ list_flow,
                            int* __restrict__ list_bdy, int* __restrict__ list_count,
                            const double* __restrict__ vt_src, double* __restrict__ vt_dst) {
    __shared__ int sh_rank[TPB / 32][64];
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = k < c.n;
    int mt = 0;
    // ascending old index inside the cell: this particle's rank among the cell's (a pass of
    // its own, one thread per cell, took 15 us on a 2D grid and 158 us on the 3D benchmark's)
    int s = 0, cb = 0, ce = 0;
    if (live) {
        s = perm[k];
        const int cell = cell_of[s];
        cb = cell_start[cell];
        ce = cell_start[cell + 1];
    }
    const bool ranks = live && ce - cb <= small;
    const int r = rank_in_cell(perm, cb, ce, s, ranks, sh_rank[threadIdx.x >> 5]);
    if (ranks) k = cb + r;
    if (live) {
        const size_t n = c.n;
        // every load before the first store: the compiler cannot tell the planes apart, and a
        // store between them makes each load wait for the one before it
        double xv[3], vv[3], x0[3], st[9], vt[3];
        ld3(xv, a.x, n, s);
        ld3(vv, a.v, n, s);
        ld3(x0, a.x0, n, s);
        const double rho = a.density[s], mass = a.mass[s], mV = a.m_V[s], pr = a.pressure[s];
        mt = a.mat_type[s];
        const int mid = a.mat_id[s], oid = a.obj_id[s], dyn = a.is_dynamic[s], id = a.id0[s];
        const long long f = cell_src[s];
        double eq = 0.0, eqp = 0.0;
        int flag = 0;
        if (SOIL) {
            ld9(st, a.stress, n, s);
            eq = a.strain_equ[s];
            eqp = a.strain_equ_p[s];
            flag = a.flag_retmap[s];
            if (vt_src) ld3(vt, vt_src, n, s);
        }
        st3(b.x, xv, n, k);
        st3(b.v, vv, n, k);
        st3(b.x0, x0, n, k);
        b.density[k] = rho;
        b.mass[k] = mass;
        b.m_V[k] = mV;
        b.pressure[k] = pr;
        if (SOIL) {
            st9(b.stress, st, n, k);
            b.strain_equ[k] = eq;
            b.strain_equ_p[k] = eqp;
            b.flag_retmap[k] = flag;
            if (vt_src) st3(vt_dst, vt, n, k);
        }
        b.mat_type[k] = mt;
        b.mat_id[k] = mid;
        b.obj_id[k] = oid;
        b.is_dynamic[k] = dyn;
        b.id0[k] = id;
        const bool flow = mt == MAT_FLUID || mt == MAT_SOIL;
        write_pos32(c, xv, flow, pos32 + k, pos32l + k);
        cell0[k] = f;
        if (flow && f >= 0 && f < c.G) cell_flow[f] = 1;
    }
    append(list_flow, list_count + 0, live && mt == c.flow_type, k);
    append(list_bdy, list_count + 1, live && (mt == MAT_DUMMY || mt == MAT_REP || mt == MAT_RIGID), k);
}

inline int nblk(long long n) { return (int)((n + TPB - 1) / TPB); }

}  // namespace

void scan_exclusive(const int* in, int* out, int n, int* tile_sum, cudaStream_t s) {
    if (n <= SCAN_ONE) {
        TSG_LAUNCH(k_scan_one, 1, SCAN_ONE_TPB, s, in, n, out);
        return;
    }
    int ntiles = (n + SCAN_TILE - 1) / SCAN_TILE;
    TSG_LAUNCH(k_tile_sums, ntiles, TPB, s, in, n, tile_sum);
    TSG_LAUNCH(k_scan_tiles, 1, TPB, s, tile_sum, ntiles);
    TSG_LAUNCH(k_tile_rescan, ntiles, TPB, s, in, n, tile_sum, out);
}

void sort_cells(int n, int nbins, const int* count, int* cell_start, int* tile_sum, const int* cell_of, const int* rank,
                int* perm, int* big, int* nbig, cudaStream_t s) {
    if (n <= SCATTER_ONE && nbins <= SCAN_ONE) {
        TSG_LAUNCH(k_scan_scatter, 1, SCAN_ONE_TPB, s, count, nbins, cell_start, n, cell_of, rank, perm);
        return;
    }
    scan_exclusive(count, cell_start, nbins, tile_sum, s);
    TSG_LAUNCH(k_scatter, nblk(n), TPB, s, n, cell_of, rank, cell_start, perm, sort_small(n), big, nbig);
    if (n > kSortAll) TSG_LAUNCH(k_cell_sort_big, 152, kSortBlock, s, big, nbig, cell_start, cell_of, n, perm);
}

void sort_fp64(const Consts& c, Persist64& cur, Persist64& nxt, Trans64& t, Grid& g, cudaStream_t s) {
    PhaseScope ph(s, PH_SORT);
    const long long nbins = c.G + 1;
    zero_async(g.count, g.zero_bytes, s);
    TSG_LAUNCH(k_hash, nblk(c.n), TPB, s, c, cur.x, g.cell_of, g.rank, g.count, g.cell0_old, g.err);
    sort_cells(c.n, (int)nbins, g.count, g.cell_start, g.tile_sum, g.cell_of, g.rank, g.perm, g.big, g.nbig, s);
    const int small = sort_small(c.n);
    // small scenes in blocks of one warp, to reach every SM
    const int tpb = c.n < 152 * 4 * TPB ? 32 : TPB, nb = (c.n + tpb - 1) / tpb;
    if (c.solver == 1) {
        TSG_LAUNCH(k_reorder64<false>, nb, tpb, s, c, g.perm, cur, nxt, t.pos32, t.pos32l, g.cell_of, g.cell_start, small, g.cell0_old,
                   t.cell0, g.cell_flow, g.list_flow, g.list_bdy, g.list_count, nullptr, nullptr);
    } else {
        // mu(I) keeps v_tmp across steps: stage it in aux3 (free until advect_pos) and gather
        const double* src = nullptr;
        if (c.solver == 2) {
            copy_async(t.aux3, t.v_tmp, sizeof(double) * 3 * (size_t)c.n, s);
            src = t.aux3;
        }
        TSG_LAUNCH(k_reorder64<true>, nb, tpb, s, c, g.perm, cur, nxt, t.pos32, t.pos32l, g.cell_of, g.cell_start, small, g.cell0_old,
                   t.cell0, g.cell_flow, g.list_flow, g.list_bdy, g.list_count, src, src ? t.v_tmp : nullptr);
    }
    Persist64 tmp = cur;
    cur = nxt;
    nxt = tmp;
}

}  // namespace tsg
