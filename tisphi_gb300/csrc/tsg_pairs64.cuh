// Neighbour rows of the FP64 form: built once per step, walked by every pair loop of it.
//
// Positions are fixed from the sort to advect_pos, so the neighbours of a step, their kernel
// gradients and the dummies' kernel values are the same in every loop.  k_list64 writes each
// particle's neighbours in the reference's traversal order (for_all_neighbors,
// eng/particle_system.py:259-269): flow particles list all neighbours, boundary and rigid
// particles only flow neighbours (all that any loop reads).  The correction pass computes the
// pair geometry and stores it beside the entries.
//
// What bounds these loops is the FP64 pipe: sm_103a issues one FP64 warp instruction per SM
// in 16 cycles, against four of any other kind per cycle, so everything that is not FP64
// arithmetic (list and record traffic, shared-memory exchange) hides behind it and every FP64
// operation saved counts.  What can leave that pipe runs on the integer pipes beside it (int_mul,
// int_sqrt, int_quot); the additions stay.  A traversal of the cells ran the FP64 body for a third of a warp's
// lanes (the candidates of different particles pass the distance test at different trips);
// rows keep the lanes full.
//
// G lanes share a row: lane g evaluates the pair terms of slots g, g + G, ..., the terms of a
// trip go through shared memory, and lane c adds component c of them in slot order.  The sums
// therefore round exactly as one thread adding them in traversal order (a missing slot adds
// +0.0, which changes no sum that starts at +0.0), C chains of additions cost the lanes
// of a row about G additions instead of C x G, and small scenes get G times the threads.
#pragma once

#include "tsg_internal.h"

namespace tsg {
namespace {

constexpr int ROWS = 32;           // rows per block; one thread each in the epilogue
constexpr int NB_BDY = 1 << 31;    // entry flag: not a flow particle (sign bit)

__device__ __forceinline__ int nb_index(int ent) { return ent & 0x7fffffff; }
__device__ __forceinline__ bool nb_flow(int ent) { return ent >= 0; }

// Distance, in cells, from coordinate t to the next cell in direction o (0: its own), or 0 where
// f32 leaves open which cell t lies in.  Coordinates below 0 truncate towards it, which only
// widens the gap.
__device__ __forceinline__ float edge(float t, int o) {
    const float f = t - floorf(t), d = o < 0 ? f : 1.f - f;
    return o != 0 && fabsf(f - 0.5f) < 0.5f - 0x1p-9f ? d : 0.f;
}

// One warp per row, or RPW rows.  The candidates of one stencil row of cells are contiguous; 32
// of them are tested at a time and the accepted ones compacted in order by ballot.  An FP64
// instruction costs a warp the same 16 cycles for one lane as for 32, so no FP64 runs here but
// for pairs within 2^-18 of R^2: the f32 distance decides all but those within 2^-10 (the
// rounding of f32 coordinates below 500 R stays under a fifth of that), the same distance with
// the low parts of the coordinates added all but those within 2^-18 (its error is below 2^-20),
// and the rest take the reference's test: r2 < R2T is sqrt(r2) < support_radius, exactly, sqrt
// being monotone.  The cell index comes from the sort (or the position refresh), one division
// per particle there instead of one per warp here.
// The pass is bound by issue, so what can be left out is: in 3D cells that lie wholly outside
// the support (a quarter of the 27; only while the cells are those of the current positions),
// and for boundary rows stencil rows without flow particles (three quarters of a tank's dummies
// see none).
// 118 k fluid + 357 k dummy particles in 3D: 210 us (294 us with all 27 cells tested, one row a
// warp and the tests of a candidate in branches; 282 with the cells left out, 226 with three
// rows a warp).  911,754 + 1,413,114: 6.34 ms with FP64 cell indices and shell tests in the warp.
template <int DIM, int RPW>
__global__ void __launch_bounds__(256) k_list64(Consts c, const double* __restrict__ X,
                                                const float4* __restrict__ P32, const float4* __restrict__ P32L,
                                                const long long* __restrict__ cell0, const int* __restrict__ cs,
                                                const unsigned char* __restrict__ cell_flow,
                                                const int* __restrict__ list_flow, int n_flow,
                                                const int* __restrict__ list_bdy, int n_bdy, bool flow_only,
                                                Pairs64 pr) {
    constexpr int NR = DIM == 3 ? 9 : 3;
    const int row0 = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * RPW, rows = n_flow + n_bdy;
    const int lane = threadIdx.x & 31;
    if (row0 >= rows) return;
    const size_t n = c.n;
    const auto near_origin = [&](const float4& p) {
        return c.pf_on && fabsf(p.x) < c.pf_lim && fabsf(p.y) < c.pf_lim && fabsf(p.z) < c.pf_lim;
    };
    // lane NR r + q: the candidates of row row0 + r in its stencil row q
    int i_l = 0, jb_l = 0, je_l = 0;
    const int row_l = row0 + lane / NR;
    if (lane < NR * RPW && row_l < rows) {
        const int q = lane % NR;
        i_l = row_l < n_flow ? list_flow[row_l] : list_bdy[row_l - n_flow];
        const long long fc = cell0[i_l];
        bool any = fc != kNoCell, below = true, above = true;
        const int ox = DIM == 3 ? q / 3 - 1 : q - 1, oy = DIM == 3 ? q % 3 - 1 : 0;
        if (DIM == 3 && cell_flow) {
            const float4 p = P32[i_l];
            if (near_origin(p)) {
                const float ex = edge(p.x * c.cell_inv, ox), ey = edge(p.y * c.cell_inv, oy);
                const float el = edge(p.z * c.cell_inv, -1), eh = edge(p.z * c.cell_inv, 1);
                const float d2 = ex * ex + ey * ey;
                any = any && !(d2 > c.cell_lim);
                below = !(d2 + el * el > c.cell_lim);
                above = !(d2 + eh * eh > c.cell_lim);
            }
        }
        if (any) {
            const long long nz = c.gnum[2], f0 = fc + ox * (c.gnum[1] * nz) + oy * nz;
            const long long f_lo = below ? f0 - 1 : f0, f_hi = above ? f0 + 1 : f0;
            const long long lo = f_lo > 0 ? f_lo : 0;
            const long long hi = f_hi < c.G - 1 ? f_hi : c.G - 1;
            any = lo <= hi;
            if (any && (row_l >= n_flow || flow_only) && cell_flow) {
                any = false;
                for (long long f = lo; f <= hi; ++f) any = any || cell_flow[f];
            }
            if (any) { jb_l = cs[lo]; je_l = cs[hi + 1]; }
        }
    }
    const unsigned some = __ballot_sync(0xffffffffu, jb_l < je_l);
    for (int r = 0; r < RPW && row0 + r < rows; ++r) {
        const int row = row0 + r;
        unsigned left = RPW == 1 ? some : (some >> (NR * r)) & ((1u << NR) - 1u);
        int m = 0;
        if (left) {
            const bool bdy = row >= n_flow, want_flow = bdy || flow_only;
            const int i = __shfl_sync(0xffffffffu, i_l, NR * r);
            const int cap = bdy ? pr.cap_b : pr.cap_f;
            int* out = bdy ? pr.nb_b + (size_t)(row - n_flow) * cap : pr.nb_f + (size_t)row * cap;
            const float4 pi = P32[i];
            const bool pf = near_origin(pi);
            const float in2 = pf ? c.pf_in2 : -1.f, out2 = pf ? c.pf_r2 : __int_as_float(0x7f800000);
            do {
                const int q = NR * r + __ffs(left) - 1;
                left &= left - 1u;
                const int jb = __shfl_sync(0xffffffffu, jb_l, q), je = __shfl_sync(0xffffffffu, je_l, q);
                for (int b = jb; b < je; b += 32) {
                    const int j = b + lane;
                    const float4 pj = P32[min(j, je - 1)];
                    const bool flow = pj.w != 0.f;
                    float fx = pi.x - pj.x, fy = pi.y - pj.y, fz = pi.z - pj.z;
                    float r2f = fx * fx + fy * fy;
                    if (DIM == 3) r2f += fz * fz;
                    bool in = j < je && j != i && (flow || !want_flow) && !(r2f > out2);
                    if (in && !(r2f < in2)) {
                        const float4 li = P32L[i], lj = P32L[j];
                        fx += li.x - lj.x;
                        fy += li.y - lj.y;
                        r2f = fx * fx + fy * fy;
                        if (DIM == 3) { fz += li.z - lj.z; r2f += fz * fz; }
                        in = pf && r2f < c.pf_lo2;
                        if (!in && !(pf && r2f > c.pf_hi2)) {
                            const double rx = X[i] - X[j], ry = X[n + i] - X[n + j];
                            double r2 = rx * rx + ry * ry;
                            if (DIM == 3) { const double rz = X[2 * n + i] - X[2 * n + j]; r2 = r2 + rz * rz; }
                            in = r2 < c.R2T;
                        }
                    }
                    const unsigned bal = __ballot_sync(0xffffffffu, in);
                    const int pos = m + __popc(bal & ((1u << lane) - 1u));
                    if (in && pos < cap) out[pos] = flow ? j : j | NB_BDY;
                    m += __popc(bal);
                }
            } while (left);
        }
        if (lane == 0) pr.cnt[row] = m;
    }
}

// FP64 products and quotients of the rare operands that the paths below leave out.  Calls, so
// that they stay behind a branch: inlined, the compiler predicates them, and an FP64 instruction
// with every lane off holds the pipe like any other.
__device__ __noinline__ double slow_mul(double a, double b) { return a * b; }
__device__ __noinline__ double slow_div(double a, double b) { return a / b; }
__device__ __noinline__ double slow_sqrt(double a) { return sqrt(a); }

// a / b, correctly rounded, from y = RN(1 / b): one product and two fused multiply-adds instead
// of the division's ten-odd FP64 instructions (Markstein 1990; Brisebarre, Muller and Raina,
// "Accelerating correctly rounded floating-point division when the divisor is known in
// advance", 2004).  The residual must not underflow nor the quotient leave the normal range:
// b is a caller's positive divisor within 2^+-200 of 1, and |a| outside [2^-500, 2^500) takes
// the division, except +-0, whose quotient is itself.
__device__ __forceinline__ double div_by(double a, double b, double y, unsigned span) {
    const unsigned hi = (unsigned)__double2hiint(a) & 0x7fffffffu;
    if (hi - (523u << 20) < span) {
        const double q = a * y;
        return __fma_rn(__fma_rn(-b, q, a), y, q);
    }
    if ((hi | (unsigned)__double2loint(a)) == 0u) return a;
    return slow_div(a, b);
}

// a * b, correctly rounded, on the integer pipes.  sm_103a issues an FP64 warp instruction per SM
// in 16 cycles; this takes about as long on the other pipes and runs beside it (measured: 18.5
// cycles at the nominal clock for the FP64 product, 15.8 for this one, 9.3 for each of two in
// parallel), so the pair loops give it most of their products.  3D, 118 k rows, us per launch:
// rates 1,835 -> 855 (first loop) and 1,476 -> 655 (second), correction 2,057 -> 1,376; with the
// roots and quotients below and the registers bounded 778, 578 and 897.  The 53 x 53 bit product of the
// significands is formed in 128 bits, normalised, and rounded to nearest even with the bits
// below jammed into one word; the sign and the exponent are put together beside it.  Operands
// are +-0 or normal numbers with normal products (usable(a), usable(b): then so are products of
// up to three of them).
__device__ __forceinline__ bool usable(double a) {  // +-0 or 2^-255 <= |a| < 2^257
    const unsigned hi = (unsigned)__double2hiint(a) & 0x7fffffffu;
    return (hi - (768u << 20) < (512u << 20)) | ((hi | (unsigned)__double2loint(a)) == 0u);
}
__device__ __forceinline__ bool zero(double a) {
    return (((unsigned)__double2hiint(a) & 0x7fffffffu) | (unsigned)__double2loint(a)) == 0u;
}
__device__ __forceinline__ double int_mul(double a, double b) {
    const unsigned ah = __double2hiint(a), al = __double2loint(a);
    const unsigned bh = __double2hiint(b), bl = __double2loint(b);
    // significands: a's in 53 bits, b's shifted up to 64
    const unsigned ma = (ah & 0xfffffu) | 0x100000u;
    const unsigned mh = __funnelshift_l(bl, bh, 11) | 0x80000000u, ml = bl << 11;
    const unsigned long long p0 = (unsigned long long)al * ml;
    const unsigned long long p1 = (unsigned long long)al * mh + (p0 >> 32);
    const unsigned long long p2 = (unsigned long long)ma * ml + (unsigned)p1;
    const unsigned long long p3 = (unsigned long long)ma * mh + (p1 >> 32) + (p2 >> 32);  // [2^51, 2^53)
    unsigned w = (unsigned)p2 | min((unsigned)p0, 1u);  // the bits below p3, the last ones jammed
    unsigned h1 = (unsigned)(p3 >> 32), h0 = (unsigned)p3;
    const unsigned sh = (h1 >> 20) ^ 1u;  // one bit short: shift up
    h1 = __funnelshift_l(h0, h1, sh);
    h0 = __funnelshift_l(w, h0, sh);
    w <<= sh;
    const unsigned up = w > 0x80000000u - (h0 & 1u);  // above half, or half and odd
    const unsigned ea = ah & 0x7ff00000u, eb = bh & 0x7ff00000u;
    const unsigned e = ea + eb - (1023u << 20) - (sh << 20) + h1;
    const unsigned long long r = (((unsigned long long)e << 32) | h0) + up;
    const bool none = min(ea, eb) == 0u;  // a zero factor
    return __hiloint2double((int)((none ? 0u : (unsigned)(r >> 32)) | ((ah ^ bh) & 0x80000000u)),
                            none ? 0 : (int)(unsigned)r);
}


// Square roots and quotients on the integer pipes, correctly rounded.  All three start from the
// f32 approximation of the special-function unit and refine it by Newton's iteration in fixed
// point on exact residuals (the low 64 bits suffice, the residuals are small); the last bit is
// then decided exactly: with M0 the truncated result and t = 2 M0 + 1 the midpoint above it,
// the sign of v - t^2 (root) or a - t b (quotient) says whether to round up.  Neither a root
// nor a quotient of 53-bit numbers is ever such a midpoint.  The tie test needs the refined
// value to a fraction of the last place only, so approximations off by a few f32 ulp give the
// same bits.
__device__ __forceinline__ unsigned approx31(float y) {  // y in (0.5, 1 + 2^-22] as 31 fractional bits
    return min(__float2uint_rz(y * 2147483648.f), 0x7fffffffu);
}
// 2^63 / B to within 2^-58 for a positive normal b = B 2^e, B in [1, 2).
__device__ __forceinline__ unsigned long long recip63(double b) {
    const unsigned bh = (unsigned)__double2hiint(b), bl = (unsigned)__double2loint(b);
    const unsigned mh = (bh & 0xfffffu) | 0x100000u;
    const unsigned long long mb = ((unsigned long long)mh << 32) | bl;
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(0x3f800000u | __funnelshift_l(bl, bh & 0xfffffu, 3))));
    const unsigned X0 = approx31(y);
    const long long R0 = (long long)(0ull - (unsigned long long)X0 * bl - ((unsigned long long)(X0 * mh) << 32));
    const unsigned long long X1 = ((unsigned long long)X0 << 32)
                                + (unsigned long long)(((long long)(int)X0 * (int)(R0 >> 32)) >> 19);
    const unsigned long long Xp = X1 >> 15;
    const long long R1 = (long long)(0ull - Xp * mb);
    return (Xp << 15) + (unsigned long long)(((long long)(int)(Xp >> 17) * (int)(R1 >> 28)) >> 40);
}
// a / b with X = recip63(b); b positive, both normal, the quotient too.
__device__ __forceinline__ double int_quot(double a, double b, unsigned long long X) {
    const unsigned ah = (unsigned)__double2hiint(a), bh = (unsigned)__double2hiint(b);
    const unsigned long long ma = ((unsigned long long)((ah & 0xfffffu) | 0x100000u) << 32) | (unsigned)__double2loint(a);
    const unsigned long long mb = ((unsigned long long)((bh & 0xfffffu) | 0x100000u) << 32) | (unsigned)__double2loint(b);
    const unsigned long long P = __umul64hi(ma << 11, X);
    const unsigned sh = (unsigned)(P >> 62) ^ 1u;  // the quotient of the significands is below one
    const unsigned long long M0 = (P << sh) >> 10;
    const long long D = (long long)((ma << (53 + sh)) - (2 * M0 + 1) * mb);
    const unsigned e = (1022u << 20) + (ah & 0x7ff00000u) - (bh & 0x7ff00000u) - (sh << 20);
    const unsigned long long r = ((unsigned long long)e << 32) + M0 + (D > 0 ? 1u : 0u);
    return __longlong_as_double((long long)(r | ((unsigned long long)(ah & 0x80000000u) << 32)));
}
// sqrt(v), v positive and normal.
__device__ __forceinline__ double int_sqrt(double v) {
    const unsigned vh = (unsigned)__double2hiint(v), vl = (unsigned)__double2loint(v);
    const int u = (int)(vh >> 20) - 1023;
    const unsigned odd = (unsigned)u & 1u;
    const unsigned long long A = ((((unsigned long long)((vh & 0xfffffu) | 0x100000u)) << 32) | vl) << odd;
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y)
        : "f"(__uint_as_float((0x3f800000u + (odd << 23)) | __funnelshift_l(vl, vh & 0xfffffu, 3))));
    const unsigned Y0 = approx31(y);
    const unsigned S0 = (unsigned)(((unsigned long long)(unsigned)(A >> 22) * Y0) >> 31);
    const long long R0 = (long long)((A << 8) - (unsigned long long)S0 * S0);
    const unsigned long long S1 = ((unsigned long long)S0 << 22)
                                + (unsigned long long)(((long long)(int)(R0 >> 12) * (int)Y0) >> 28);
    const unsigned long long Sp = S1 >> 8;
    const long long R1 = (long long)((A << 36) - Sp * Sp);
    const unsigned long long M0 = (Sp << 8) + (unsigned long long)(((long long)(int)(R1 >> 20) * (int)Y0) >> 48);
    const unsigned long long t = 2 * M0 + 1;
    const long long D = (long long)((A << 54) - t * t);
    return __longlong_as_double((long long)(((unsigned long long)(unsigned)(1022 + (u >> 1)) << 52) + M0 + (D > 0 ? 1u : 0u)));
}
// A divisor prepared for int_quot (0: not usable, quotients take the call).
__device__ __forceinline__ unsigned long long divisor(double b) {  // usable: 2^-200 <= b < 2^200
    return (unsigned)__double2hiint(b) - (823u << 20) < 400u << 20 ? recip63(b) : 0ull;
}

// a > b for b >= 0 and a that is not a NaN, on the bits (an FP64 comparison holds the pipe too).
__device__ __forceinline__ bool above(double a, double b) {
    return __double_as_longlong(a) > __double_as_longlong(b);
}

// fmin(x, 0.0) without an FP64 comparison: x where its sign is set (and it is no NaN), else 0.
__device__ __forceinline__ double min0(double x) {
    const int hi = __double2hiint(x), lo = __double2loint(x);
    const bool keep = hi < 0 && ((unsigned)hi < 0xfff00000u || ((unsigned)hi == 0xfff00000u && lo == 0));
    return keep ? x : 0.0;
}

// Flattened cell index (truncating cast, eng/particle_system.py:216-226), unclipped; kNoCell
// where a coordinate leaves the int range or is not finite.
__device__ __forceinline__ long long flat_cell(const Consts& c, const double* x) {
    long long idx[3];
    for (int d = 0; d < 3; ++d) {
        const double t = div_by(x[d] - c.vs[d], c.grid, c.rgrid, c.grid_span);
        if (!(fabs(t) < 2147483647.0)) return kNoCell;
        idx[d] = (long long)(int)t;
    }
    return idx[0] * c.gnum[1] * c.gnum[2] + idx[1] * c.gnum[2] + idx[2];
}

// Planar vectors and tensors.
__device__ __forceinline__ void ld3(double* r, const double* a, size_t n, int i) {
#pragma unroll
    for (int d = 0; d < 3; ++d) r[d] = a[d * n + i];
}
__device__ __forceinline__ void st3(double* a, const double* r, size_t n, int i) {
#pragma unroll
    for (int d = 0; d < 3; ++d) a[d * n + i] = r[d];
}
__device__ __forceinline__ void ld9(double* r, const double* a, size_t n, int i) {
#pragma unroll
    for (int q = 0; q < 9; ++q) r[q] = a[q * n + i];
}
__device__ __forceinline__ void st9(double* a, const double* r, size_t n, int i) {
#pragma unroll
    for (int q = 0; q < 9; ++q) a[q * n + i] = r[q];
}
// f32 coordinates of a position: high part (w: flow flag) and what it rounds off.
__device__ __forceinline__ void write_pos32(const Consts& c, const double* x, bool flow, float4* hi, float4* lo) {
    double d[3];
    float h[3];
    for (int q = 0; q < 3; ++q) { d[q] = x[q] - c.vs[q]; h[q] = (float)d[q]; }
    *hi = make_float4(h[0], h[1], h[2], flow ? 1.f : 0.f);
    *lo = make_float4((float)(d[0] - h[0]), (float)(d[1] - h[1]), (float)(d[2] - h[2]), 0.f);
}

// The ordered sums of one row's C pair terms by its G lanes; acc[m] of lane g is component
// g + m G.  `term(s, T)` evaluates slot s.  sh: this warp's C x 33 doubles (the pitch keeps
// the column reads off each other's banks).
template <int C, int G, class F>
__device__ __forceinline__ void row_sums(int cnt, double* sh, double (&acc)[(C + G - 1) / G], F&& term) {
    const int lane = threadIdx.x & 31, g = lane % G, gb = lane - g;
    const int mx = __reduce_max_sync(0xffffffffu, cnt);
    for (int k0 = 0; k0 < mx; k0 += G) {
        double T[C];
#pragma unroll
        for (int q = 0; q < C; ++q) T[q] = 0.0;
        if (k0 + g < cnt) term(k0 + g, T);
#pragma unroll
        for (int q = 0; q < C; ++q) sh[q * 33 + lane] = T[q];
        __syncwarp();
#pragma unroll
        for (int m = 0; m < (C + G - 1) / G; ++m) {
            const int q = g + m * G;
            if (q < C) {
#pragma unroll
                for (int e = 0; e < G; ++e) acc[m] = acc[m] + sh[q * 33 + gb + e];
            }
        }
        __syncwarp();
    }
}

// Row sums of a block of ROWS rows: fills S[q][row in block] (shared) for every listed row.
// cnt is this thread's row's count, 0 for rows to skip.  Ends with a block barrier.
template <int C, int G, class F>
__device__ __forceinline__ void block_row_sums(int cnt, double (*S)[ROWS], F&& term) {
    __shared__ double sh[G][C * 33];
    double acc[(C + G - 1) / G];
#pragma unroll
    for (int m = 0; m < (C + G - 1) / G; ++m) acc[m] = 0.0;
    row_sums<C, G>(cnt, sh[threadIdx.x >> 5], acc, term);
    const int g = threadIdx.x % G, r = threadIdx.x / G;
#pragma unroll
    for (int m = 0; m < (C + G - 1) / G; ++m)
        if (g + m * G < C) S[g + m * G][r] = acc[m];
    __syncthreads();
}

}  // namespace
}  // namespace tsg
