// FP64 form of the per-substep SPH path (the "plain FP64" GPU form).
//
// Every arithmetic expression follows the reference's evaluation order (Python/Taichi
// left-to-right; sums over neighbours in for_all_neighbors order, eng/particle_system.py:
// 259-269), and this file is compiled with -fmad=false, so with IEEE f64 division and
// square root the results are bit-identical to the f64 CPU oracle.  Constant powers are
// products: q1^4 = (q1*q1)*(q1*q1), q1^3 = (q1*q1)*q1, x**2 = x*x.
//
// Kernels (one thread per particle; boundary / flow particles through index lists):
//   k_corr_flow, k_corr_bdy  Shepard factor for all particles, CSPM matrix for flow particles
//                 (eng/solver_sph_base.py:386-423), pair geometry of the rows.
//   k_particle    the per-particle passes: init_real2tmp (eng/solver_sph_base.py:67-74), the
//                 first phase of one_step (Tait EOS, eng/solver_sph_wc.py:86-88, or stress
//                 adaptation, eng/solver_sph_dp.py:215-217), the integrators, advect_pos and
//                 the solvers' post-steps (eng/solver_sph_base.py:79-247, solver overrides).
//   k_bdy         dummy-boundary extrapolation of v_tmp, density_tmp, pressure / stress
//                 (eng/solver_sph_wc.py:90-103, eng/solver_sph_muI.py:97-109,
//                 eng/solver_sph_dp.py:219-234), all sums in one traversal.
//   k_wc_rates    continuity + momentum (eng/solver_sph_wc.py:108-126), one traversal.
//   k_mui_stress  mu(I) velocity gradient, continuity, stress (eng/solver_sph_muI.py:67-92).
//   k_mui_mom     mu(I) stress divergence + damping (eng/solver_sph_muI.py:113-128).
//   k_dp_rates    DP velocity gradient, continuity, Bui-2008 stress rate, stress
//                 divergence, damping (eng/solver_sph_dp.py:236-270), one traversal.
#include <cfloat>

#include "tsg_internal.h"
#include "tsg_pairs64.cuh"
#include "tsg_polar.cuh"
#include "tsg_rigid_list.cuh"

namespace tsg {

namespace {

constexpr int TPB = 128;

inline int nblk(long long n, int tpb = TPB) { return (int)((n + tpb - 1) / tpb); }

// ---- kernel functions (eng/solver_sph_base.py:299-358) ----
// W and |grad W| factor from the precomputed norm rn; dW_c = s * r_c / rn (Wendland) or
// s * (r_c / rn * h1) (cubic), matching the reference's expression trees.
template <class P>
__device__ __forceinline__ double kernel_W(const P& c, double rn) {
    double res = 0.0;
    double q = rn * c.h1;
    if (rn > EPS && q <= 2.0) {
        if (c.kernel == 1) {
            double q1 = __fma_rn(-0.5, q, 1.0);  // 0.5 q and 2 q are exact: one rounding either way
            res = c.kk * ((q1 * q1) * (q1 * q1)) * __fma_rn(2.0, q, 1.0);
        } else if (q <= 1.0) {
            double q2 = q * q, q3 = q2 * q;
            res = c.kk * (0.5 * q3 - q2 + 2.0 / 3.0);
        } else {
            double t = 2.0 - q;
            res = c.kk / 6.0 * ((t * t) * t);
        }
    }
    return res;
}

template <int DIM, class P>
__device__ __forceinline__ void kernel_dW(const P& c, const double* r, double rn, double* out) {
    out[0] = out[1] = out[2] = 0.0;
    double q = rn * c.h1;
    if (rn > EPS && q <= 2.0) {
        const double y = __drcp_rn(rn);
        if (c.kernel == 1) {
            double q1 = __fma_rn(-0.5, q, 1.0);
            double s = c.kk * ((q1 * q1) * q1) * (-5.0 * q) * c.h1;
            for (int d = 0; d < DIM; ++d) out[d] = div_by(s * r[d], rn, y, c.div_span);
        } else {
            double s;
            if (q <= 1.0) s = c.kk * q * (1.5 * q - 2.0);
            else { double f = 2.0 - q; s = c.kk * (-0.5 * f * f); }
            for (int d = 0; d < DIM; ++d) out[d] = s * (div_by(r[d], rn, y, c.div_span) * c.h1);
        }
    }
}

template <int DIM, class M>
__device__ __forceinline__ void matvec_corr(const double* L, const double* k, double* out, M mul) {
    for (int p = 0; p < DIM; ++p) {
        double s = mul(L[3 * p], k[0]) + mul(L[3 * p + 1], k[1]);
        if (DIM == 3) s = s + mul(L[3 * p + 2], k[2]);
        out[p] = s;
    }
    if (DIM == 2) out[2] = 0.0;
}

template <int DIM, class M>
__device__ __forceinline__ double dotv(const double* a, const double* b, M mul) {
    double s = mul(a[0], b[0]) + mul(a[1], b[1]);
    if (DIM == 3) s = s + mul(a[2], b[2]);
    return s;
}
// The pipe of a run of products: integer where every operand is usable, else calls.
struct IntMul { __device__ __forceinline__ double operator()(double a, double b) const { return int_mul(a, b); } };
struct SlowMul { __device__ __forceinline__ double operator()(double a, double b) const { return slow_mul(a, b); } };
struct PlainMul { __device__ __forceinline__ double operator()(double a, double b) const { return a * b; } };
template <class F>
__device__ __forceinline__ void on_pipe(bool usable_operands, F&& f) {
    if (usable_operands) f(IntMul());
    else f(SlowMul());
}
struct IntQuot {
    __device__ __forceinline__ double operator()(double a, double b, unsigned long long X) const {
        const double q = int_quot(a, b, X);
        return zero(a) ? a : q;
    }
};
struct SlowQuot {
    __device__ __forceinline__ double operator()(double a, double b, unsigned long long) const { return slow_div(a, b); }
};
struct Check {
    bool& ok;
    __device__ __forceinline__ void operator()(double x) const { ok = ok & usable(x); }
    __device__ __forceinline__ void operator()(bool cond) const { ok = ok & cond; }
    template <int N>
    __device__ __forceinline__ void all(const double* x) const {
#pragma unroll
        for (int q = 0; q < N; ++q) ok = ok & usable(x[q]);
    }
};
struct NoCheck {
    __device__ __forceinline__ void operator()(double) const {}
    __device__ __forceinline__ void operator()(bool) const {}
    template <int N>
    __device__ __forceinline__ void all(const double*) const {}
};
// eval(mul, quot, check) evaluates a pair's terms and names every operand that the integer
// routines must be able to use; they return garbage (no fault, no loop) for others, so the terms
// are formed first, without a branch, and once more by the FP64 unit where a check failed.  A
// branch before each run of products kept the compiler from overlapping their chains.
template <class E>
__device__ __forceinline__ void on_pipes(E&& eval) {
    bool ok = true;
    eval(IntMul(), IntQuot(), Check{ok});
    if (!ok) eval(SlowMul(), SlowQuot(), NoCheck());
}
// Every entry usable by int_mul.
template <int DIM>
__device__ __forceinline__ bool usable_v(const double* a) {
    return usable(a[0]) & usable(a[1]) & (DIM == 2 || usable(a[2]));
}
template <int DIM>
__device__ __forceinline__ bool usable_m(const double* L) {
    bool ok = true;
    for (int a = 0; a < DIM; ++a)
        for (int b = 0; b < DIM; ++b) ok = ok && usable(L[3 * a + b]);
    return ok;
}

// ---- neighbour traversal (eng/particle_system.py:259-269) ----
// Visits the 3^dim cells around the centre's cell in ndrange order (z fastest); the three
// cells of one row have consecutive flattened indices, so each row is one contiguous index
// range (the reference's flattening, aliasing included).  Rows are clipped to [0, G).
// A candidate is a neighbour when j != i and sqrt(|x_i - x_j|^2) < support_radius in f64;
// the f32 prefilter only rejects candidates that are certainly farther away.
template <int DIM, class F>
__device__ __forceinline__ void for_neighbors(const Consts& c, const double* __restrict__ X,
                                              const float4* __restrict__ P32, const int* __restrict__ cs,
                                              int i, const double* xi, bool prefilter, F&& body) {
    const int n = c.n;
    long long cc[3];
    for (int d = 0; d < 3; ++d) {
        double t = (xi[d] - c.vs[d]) / c.grid;
        if (!(fabs(t) < 2147483647.0)) return;
        cc[d] = (int)t;
    }
    const long long ny = c.gnum[1], nz = c.gnum[2], G = c.G;
    float4 pi = make_float4(0.f, 0.f, 0.f, 0.f);
    bool pf = prefilter && c.pf_on;
    if (pf) {
        pi = P32[i];
        pf = fabsf(pi.x) < c.pf_lim && fabsf(pi.y) < c.pf_lim && fabsf(pi.z) < c.pf_lim;
    }
#pragma unroll 1
    for (int ox = -1; ox <= 1; ++ox) {
#pragma unroll 1
        for (int oy = (DIM == 3 ? -1 : 0); oy <= (DIM == 3 ? 1 : 0); ++oy) {
            long long f0 = (cc[0] + ox) * ny * nz + (cc[1] + oy) * nz + cc[2];
            long long lo = f0 - 1 > 0 ? f0 - 1 : 0;
            long long hi = f0 + 1 < G - 1 ? f0 + 1 : G - 1;
            if (lo > hi) continue;
            const int jb = cs[lo], je = cs[hi + 1];
#pragma unroll 1
            for (int j = jb; j < je; ++j) {
                if (j == i) continue;
                if (pf) {
                    float4 pj = P32[j];
                    float fx = pi.x - pj.x, fy = pi.y - pj.y, fz = pi.z - pj.z;
                    float r2f = fx * fx + fy * fy;
                    if (DIM == 3) r2f += fz * fz;
                    if (r2f > c.pf_r2) continue;
                }
                double r[3];
                r[0] = xi[0] - X[j];
                r[1] = xi[1] - X[(size_t)n + j];
                r[2] = DIM == 3 ? xi[2] - X[2 * (size_t)n + j] : 0.0;
                double r2 = r[0] * r[0] + r[1] * r[1];
                if (DIM == 3) r2 = r2 + r[2] * r[2];
                double rn = sqrt(r2);
                if (!(rn < c.R)) continue;
                body(j, r, rn);
            }
        }
    }
}

template <int DIM>
__device__ __forceinline__ void load_x(const double* X, int i, int n, double* xi) {
    xi[0] = X[i];
    xi[1] = X[(size_t)n + i];
    xi[2] = DIM == 3 ? X[2 * (size_t)n + i] : X[2 * (size_t)n + i];
}

__device__ __forceinline__ bool is_flow(int t) { return t == MAT_FLUID || t == MAT_SOIL; }

// ---- CSPM (eng/solver_sph_base.py:386-423) ----
__device__ __forceinline__ double det2(const double* a) { return a[0] * a[4] - a[1] * a[3]; }
__device__ __forceinline__ double det3(const double* a) {
    return a[0] * (a[4] * a[8] - a[7] * a[5]) - a[3] * (a[1] * a[8] - a[7] * a[2]) + a[6] * (a[1] * a[5] - a[4] * a[2]);
}

// The kernel functions behind a call (see slow_mul), their constants by value: grad W and W.
struct KernelConsts { int kernel; unsigned div_span; double h1, kk; };
struct KernelVals { double kd[3], W, rr; };  // grad W, W, |r| |r|
template <int DIM>
__device__ __noinline__ KernelVals slow_kernel(KernelConsts c, double r0, double r1, double r2, double rn) {
    const double r[3] = {r0, r1, r2};
    KernelVals k;
    kernel_dW<DIM>(c, r, rn, k.kd);
    k.W = kernel_W(c, rn);
    k.rr = rn * rn;
    return k;
}

// grad W (DW) and W (WV) of a separation r.  Both kernels away from their ends run on the
// integer pipes but for their sums; separations at the ends take the kernel functions.
template <int DIM, bool DW, bool WV>
__device__ __forceinline__ KernelVals pair_kernel(const Consts& c, const double* r) {
    KernelVals k;
    k.W = 0.0;
    const double r2 = dotv<DIM>(r, r, IntMul());
    const double rn = int_sqrt(r2);
    const double q = int_mul(rn, c.h1);
    // 1 - q / 2 (Wendland) or 2 - q (cubic) must not vanish
    const double q1 = c.kernel == 1 ? __fma_rn(-0.5, q, 1.0) : 2.0 - q;
    const bool ok = (c.kern_int != 0) & usable_v<DIM>(r) & above(r2, 0x1p-200) & above(rn, EPS) & !above(q, 2.0) &
                    above(q1, 0x1p-50);
    const unsigned long long X = DW ? recip63(rn) : 0ull;
    if (DW) k.rr = int_mul(rn, rn);
    if (c.kernel == 1) {
        const double q2 = int_mul(q1, q1);
        if (DW) {
            const double s = int_mul(int_mul(int_mul(c.kk, int_mul(q2, q1)), int_mul(-5.0, q)), c.h1);
            for (int d = 0; d < DIM; ++d) k.kd[d] = IntQuot()(int_mul(s, r[d]), rn, X);
        }
        if (WV) k.W = int_mul(int_mul(c.kk, int_mul(q2, q2)), __fma_rn(2.0, q, 1.0));
    } else {
        double s, w;
        if (!above(q, 1.0)) {
            const double q2 = int_mul(q, q);
            w = int_mul(c.kk, __fma_rn(0.5, int_mul(q2, q), -q2) + 2.0 / 3.0);
            s = int_mul(int_mul(c.kk, q), int_mul(1.5, q) - 2.0);
        } else {
            w = int_mul(c.kk6, int_mul(int_mul(q1, q1), q1));
            s = int_mul(c.kk, int_mul(int_mul(-0.5, q1), q1));
        }
        if (DW)
            for (int d = 0; d < DIM; ++d) k.kd[d] = int_mul(s, int_mul(IntQuot()(r[d], rn, X), c.h1));
        if (WV) k.W = w;
    }
    if (!ok) {
        const double d2 = dotv<DIM>(r, r, SlowMul());
        k = slow_kernel<DIM>(KernelConsts{c.kernel, c.div_span, c.h1, c.kk}, r[0], r[1], r[2], slow_sqrt(d2));
    }
    return k;
}

// Pair geometry of row slot `slot` (entry j): r, grad W and, for a flow neighbour, W into
// registers, grad W and the viscosity denominator into the row's planes.  The Wendland kernel
// away from its ends runs its products on the integer pipes; the others take the kernel functions.
template <int DIM, bool WV>
__device__ __forceinline__ double pair_geometry(const Consts& c, const double* __restrict__ X, const double* xi, int j,
                                                const Pairs64& pr, size_t slot, double* r, double* kd) {
    const size_t n = c.n;
    r[0] = xi[0] - X[j];
    r[1] = xi[1] - X[n + j];
    r[2] = DIM == 3 ? xi[2] - X[2 * n + j] : 0.0;
    const KernelVals k = pair_kernel<DIM, true, WV>(c, r);
    for (int d = 0; d < DIM; ++d) {
        kd[d] = k.kd[d];
        pr.gk[d * pr.slots_f + slot] = kd[d];
    }
    if (pr.gden) {
        const double den = k.rr + c.eps_h2;
        pr.gden[slot] = make_double2(den, __longlong_as_double((long long)divisor(den)));
    }
    return k.W;
}

// Kernel value of a boundary row's entry.
template <int DIM>
__device__ __forceinline__ double pair_W(const Consts& c, const double* __restrict__ X, const double* xi, int j) {
    const size_t n = c.n;
    const double r[3] = {xi[0] - X[j], xi[1] - X[n + j], DIM == 3 ? xi[2] - X[2 * n + j] : 0.0};
    return pair_kernel<DIM, false, true>(c, r).W;
}

// This thread's row in the row-sum phase: particle index and listed count (0 for a row past the
// end or above the pitch, which the epilogue walks through the cells).
struct RowRef { int row, i, cnt; size_t base; };
template <int G>
__device__ __forceinline__ RowRef row_ref(const int* __restrict__ list, int count, const int* __restrict__ cnt, int cap) {
    RowRef q;
    q.row = blockIdx.x * ROWS + threadIdx.x / G;
    const bool live = q.row < count;
    q.i = live ? list[q.row] : list[0];
    q.cnt = live ? cnt[q.row] : 0;
    if (q.cnt > cap) q.cnt = 0;
    q.base = (size_t)q.row * cap;
    return q;
}

// Flow rows: pair geometry, Shepard sum and CSPM matrix (eng/solver_sph_base.py:386-423).
// Bounded to 80-odd registers: 24 warps an SM instead of 16 hide the integer chains (3D, 118 k
// rows: 979 -> 893 us; 2D, 7.2 k rows: 11 us a step); the 3D rates passes likewise (642 -> 585
// and 835 -> 798 us).  What holds them now is the FP64 pipe, about 80 % busy.
template <int DIM, int G, bool CORR>
__global__ void __launch_bounds__(ROWS * G, G == 8 ? 3 : 6) k_corr_flow(Consts c, Persist64 p, Trans64 t, const int* __restrict__ cs,
                                                        const int* __restrict__ list, int count, Pairs64 pr) {
    constexpr int C = 1 + (CORR ? DIM * DIM : 0);
    __shared__ double S[C][ROWS];
    const int n = c.n;
    if (pr.cap_f) {
        const RowRef q = row_ref<G>(list, count, pr.cnt, pr.cap_f);
        double xi[3];
        load_x<DIM>(p.x, q.i, n, xi);
        block_row_sums<C, G>(q.cnt, S, [&](int s, double* T) {
            const int ent = pr.nb_f[q.base + s], j = nb_index(ent);
            double r[3], kd[3];
            // a boundary neighbour adds nothing: zero mass gives +-0 terms
            const double mVj = nb_flow(ent) ? p.m_V[j] : 0.0;
            const double W = pair_geometry<DIM, true>(c, p.x, xi, j, pr, q.base + s, r, kd);
            double av[3];
            on_pipes([&](auto mul, auto, auto check) {
                check(mVj);
                check(W);
                T[0] = mul(mVj, W);
                if (CORR) {
                    check.template all<DIM>(r);
                    for (int a = 0; a < DIM; ++a) av[a] = mul(mVj, -r[a]);
                }
            });
            // (the matrix products stay on the FP64 pipe, which this pass no longer fills)
            if (CORR)
                for (int a = 0; a < DIM; ++a)
                    for (int b = 0; b < DIM; ++b) T[1 + a * DIM + b] = av[a] * kd[b];
        });
    }
    const int row = blockIdx.x * ROWS + threadIdx.x;
    if (threadIdx.x >= ROWS || row >= count) return;
    const int i = list[row];
    double s = 0.0;
    double L[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    if (pr.cap_f && pr.cnt[row] <= pr.cap_f) {
        s = S[0][threadIdx.x];
        if (CORR)
            for (int a = 0; a < DIM; ++a)
                for (int b = 0; b < DIM; ++b) L[3 * a + b] = S[1 + a * DIM + b][threadIdx.x];
    } else {
        double xi[3];
        load_x<DIM>(p.x, i, n, xi);
        for_neighbors<DIM>(c, p.x, t.pos32, cs, i, xi, true, [&](int j, const double* r, double rn) {
            if (!is_flow(p.mat_type[j])) return;
            const double mVj = p.m_V[j];
            s += mVj * kernel_W(c, rn);
            if (CORR) {
                double k[3];
                kernel_dW<DIM>(c, r, rn, k);
                for (int a = 0; a < DIM; ++a) {
                    double av = mVj * (-r[a]);
                    for (int b = 0; b < DIM; ++b) L[3 * a + b] = L[3 * a + b] + av * k[b];
                }
            }
        });
    }
    t.CSPM_f[i] = s != 0.0 ? 1.0 / s : 1.0;
    if (CORR) {
        double inv[9] = {1, 0, 0, 0, 1, 0, 0, 0, 1};
        if (DIM == 2) {
            double dt = det2(L);
            if (fabs(dt) > EPS) {
                double id = 1.0 / dt;
                inv[0] = id * L[4]; inv[1] = id * (-L[1]); inv[2] = 0.0;
                inv[3] = id * (-L[3]); inv[4] = id * L[0]; inv[5] = 0.0;
                inv[6] = 0.0; inv[7] = 0.0; inv[8] = 0.0;
            }
        } else {
            double dt = det3(L);
            if (fabs(dt) > EPS) {
                double id = 1.0 / dt;
                for (int a = 0; a < 3; ++a)
                    for (int b = 0; b < 3; ++b)
                        inv[3 * b + a] = id * (L[3 * ((a + 1) % 3) + (b + 1) % 3] * L[3 * ((a + 2) % 3) + (b + 2) % 3]
                                             - L[3 * ((a + 2) % 3) + (b + 1) % 3] * L[3 * ((a + 1) % 3) + (b + 2) % 3]);
            }
        }
        for (int q = 0; q < 9; ++q) t.CSPM_L[(size_t)q * n + i] = inv[q];
    }
}

// Boundary and rigid rows: kernel values and Shepard sum over the flow neighbours.
template <int DIM, int G>
__global__ void __launch_bounds__(ROWS * G) k_corr_bdy(Consts c, Persist64 p, Trans64 t, const int* __restrict__ cs,
                                                       const int* __restrict__ list, int count, Pairs64 pr) {
    __shared__ double S[1][ROWS];
    const int n = c.n;
    const int* cnt = pr.cnt + c.n_flow;
    if (pr.cap_f) {
        const RowRef q = row_ref<G>(list, count, cnt, pr.cap_b);
        double xi[3];
        load_x<DIM>(p.x, q.i, n, xi);
        block_row_sums<1, G>(q.cnt, S, [&](int s, double* T) {
            const int j = pr.nb_b[q.base + s];
            const double w = pair_W<DIM>(c, p.x, xi, j);
            pr.gw[q.base + s] = w;
            T[0] = p.m_V[j] * w;
        });
    }
    const int row = blockIdx.x * ROWS + threadIdx.x;
    if (threadIdx.x >= ROWS || row >= count) return;
    const int i = list[row];
    double s = 0.0;
    if (pr.cap_f && cnt[row] <= pr.cap_b) {
        s = S[0][threadIdx.x];
    } else {
        double xi[3];
        load_x<DIM>(p.x, i, n, xi);
        for_neighbors<DIM>(c, p.x, t.pos32, cs, i, xi, true, [&](int j, const double*, double rn) {
            if (is_flow(p.mat_type[j])) s += p.m_V[j] * kernel_W(c, rn);
        });
    }
    t.CSPM_f[i] = s != 0.0 ? 1.0 / s : 1.0;
    if (c.corr == 1)
        for (int q = 0; q < 9; ++q) t.CSPM_L[(size_t)q * n + i] = q % 4 == 0 ? 1.0 : 0.0;
}

// The pair geometry alone, for one_step called without the step sequence around it.
template <int DIM, int G>
__global__ void __launch_bounds__(ROWS * G) k_geom_flow(Consts c, Persist64 p, const int* __restrict__ list, int count,
                                                        Pairs64 pr) {
    const RowRef q = row_ref<G>(list, count, pr.cnt, pr.cap_f);
    double xi[3], r[3], kd[3];
    load_x<DIM>(p.x, q.i, c.n, xi);
    for (int s = threadIdx.x % G; s < q.cnt; s += G)
        pair_geometry<DIM, false>(c, p.x, xi, nb_index(pr.nb_f[q.base + s]), pr, q.base + s, r, kd);
}

template <int DIM, int G>
__global__ void __launch_bounds__(ROWS * G) k_geom_bdy(Consts c, Persist64 p, const int* __restrict__ list, int count,
                                                       Pairs64 pr) {
    const RowRef q = row_ref<G>(list, count, pr.cnt + c.n_flow, pr.cap_b);
    double xi[3];
    load_x<DIM>(p.x, q.i, c.n, xi);
    for (int s = threadIdx.x % G; s < q.cnt; s += G)
        pr.gw[q.base + s] = pair_W<DIM>(c, p.x, xi, pr.nb_b[q.base + s]);
}

// Density summation: calc_density_task summed over for_all_neighbors
// (eng/solver_sph_wc.py:30-31, eng/particle_system.py:259-269), sum_j mass_j W(x_i - x_j)
// over the neighbours j != i of every particle, in traversal order.
template <int DIM>
__global__ void k_density_sum(Consts c, Persist64 p, Trans64 t, const int* __restrict__ cs, double* __restrict__ out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    double xi[3];
    load_x<DIM>(p.x, i, c.n, xi);
    double ret = 0.0;
    for_neighbors<DIM>(c, p.x, t.pos32, cs, i, xi, true, [&](int j, const double*, double rn) {
        ret += p.mass[j] * kernel_W(c, rn);
    });
    out[i] = ret;
}

// ---- Drucker-Prager invariants and return mapping (eng/solver_sph_dp.py:42-109) ----
__device__ __forceinline__ double mtrace(const double* a) { return (a[0] + a[4]) + a[8]; }
__device__ __forceinline__ double msum_sq(const double* a) {
    double s = a[0] * a[0];
    for (int k = 1; k < 9; ++k) s = s + a[k] * a[k];
    return s;
}
__device__ __forceinline__ double msum_prod(const double* a, const double* b) {
    double s = a[0] * b[0];
    for (int k = 1; k < 9; ++k) s = s + a[k] * b[k];
    return s;
}
__device__ __forceinline__ void dp_inv(const Consts& c, const double* st, double* s, double& I1, double& sJ2, double& f) {
    double t3 = mtrace(st) / 3.0;
    for (int k = 0; k < 9; ++k) s[k] = st[k] - t3 * ((k % 4 == 0) ? 1.0 : 0.0);
    I1 = mtrace(st);
    sJ2 = sqrt(0.5 * msum_sq(s));
    f = sJ2 + c.alpha * I1 - c.k_c;
}
__device__ __forceinline__ void dp_adapt(const Consts& c, double* st) {
    double s[9], I1, sJ2, f;
    dp_inv(c, st, s, I1, sJ2, f);
    if (f > EPS_F) {
        if (f > sJ2) {
            double tt = (I1 - c.kc_over_alpha) / 3.0;
            for (int k = 0; k < 9; ++k) st[k] = st[k] - tt * ((k % 4 == 0) ? 1.0 : 0.0);
        }
        dp_inv(c, st, s, I1, sJ2, f);
        double r = (-I1 * c.alpha + c.k_c) / sJ2;
        for (int k = 0; k < 9; ++k) st[k] = r * s[k] + (((k % 4 == 0) ? 1.0 : 0.0) * I1) / 3.0;
    }
}
__device__ __forceinline__ int dp_flag(const Consts& c, const double* st) {
    double s[9], I1, sJ2, f;
    dp_inv(c, st, s, I1, sJ2, f);
    int flag = 1;
    if (f < -EPS_F) flag = 0;
    else if (f > EPS_F) flag = (f >= sJ2) ? 3 : 2;
    return flag;
}

__device__ __forceinline__ double powi(double x, long n) {
    double r = 1.0;
    bool first = true;
    while (n > 0) {
        if (n & 1) { r = first ? x : r * x; first = false; }
        n >>= 1;
        if (n) x = x * x;
    }
    return r;
}

// What the rates loop reads of a neighbour, one aligned record per particle (the expressions
// of the pair terms that depend on the neighbour alone, rounded as they are there):
//   WCSPH  v~ (3), p / (rho~ rho~), m_V, viscosity factor, -rho0 m_V, 0
//   soil   2D: v~ (2), m_V, m_V rho~, stress~ / (rho~ rho~) (xx, xy, yx, yy)
//          3D: v~ (3), m_V, m_V rho~, the nine stress entries, 0, 0
// The viscosity factor is visc_fac m_V for a fluid neighbour and (visc_fac m_V) rho0 for the
// others (eng/solver_sph_wc.py:47-62).
__device__ __forceinline__ void wc_record(const Consts& c, double* rec, int i, const double* vt, double pr, double rt,
                                          double mV, bool fluid) {
    double2* o = reinterpret_cast<double2*>(rec + (size_t)8 * i);
    const double vf = c.visc_fac * mV;
    o[0] = make_double2(vt[0], vt[1]);
    o[1] = make_double2(vt[2], pr / (rt * rt));
    o[2] = make_double2(mV, fluid ? vf : vf * c.rho0);
    o[3] = make_double2(-c.rho0 * mV, 0.0);
}
__device__ __forceinline__ void soil_record(const Consts& c, double* rec, int i, const double* vt, const double* st,
                                            double rt, double mV) {
    const double r2 = rt * rt;
    if (c.dim == 2) {
        double2* o = reinterpret_cast<double2*>(rec + (size_t)8 * i);
        o[0] = make_double2(vt[0], vt[1]);
        o[1] = make_double2(mV, mV * rt);
        o[2] = make_double2(st[0] / r2, st[1] / r2);
        o[3] = make_double2(st[3] / r2, st[4] / r2);
    } else {
        double2* o = reinterpret_cast<double2*>(rec + (size_t)16 * i);
        o[0] = make_double2(vt[0], vt[1]);
        o[1] = make_double2(vt[2], mV);
        o[2] = make_double2(mV * rt, st[0] / r2);
        for (int q = 0; q < 4; ++q) o[3 + q] = make_double2(st[1 + 2 * q] / r2, st[2 + 2 * q] / r2);
        o[7] = make_double2(0.0, 0.0);
    }
}

// One flow neighbour's terms of the dummy extrapolation: v (DIM), then p (WCSPH) or density (1)
// and stress (9).  w = W(r), r = x_i - x_j.
template <int DIM, bool SOIL>
__device__ __forceinline__ void bdy_terms(const Consts& c, const Persist64& p, const Trans64& t, int j,
                                          const double* r, double w, double* T) {
    const size_t n = c.n;
    const double mVj = p.m_V[j], rtj = t.density_tmp[j];
    for (int d = 0; d < DIM; ++d) T[d] = mVj * t.v_tmp[d * n + j] * w;
    if (!SOIL) {
        T[DIM] = mVj * (p.pressure[j] + rtj * c.g[1] * r[1]) * w;
    } else {
        T[DIM] = c.solver == 2 ? mVj * rtj * w : 0.0;
        for (int a = 0; a < 3; ++a)
            for (int b = 0; b < 3; ++b) {
                double m = t.stress_tmp[(size_t)(3 * a + b) * n + j];
                if (a == b) m = m + (rtj * c.g[a]) * r[a];
                else m = m + (rtj * 0.0) * 0.0;
                T[DIM + 1 + 3 * a + b] = mVj * m * w;
            }
    }
}

// Dummy-boundary extrapolation (Adami 2012 style), one walk of the row for every sum.
template <int DIM, int G, bool SOIL>
__global__ void __launch_bounds__(ROWS * G) k_bdy(Consts c, Persist64 p, Trans64 t, const int* __restrict__ cs,
                                                  const int* __restrict__ list, int count, Pairs64 pr) {
    constexpr int C = DIM + 1 + (SOIL ? 9 : 0);
    __shared__ double S[C][ROWS];
    const int n = c.n;
    const int* cnt = pr.cnt + c.n_flow;
    if (pr.cap_f) {
        const RowRef q = row_ref<G>(list, count, cnt, pr.cap_b);
        double xi[3];
        load_x<DIM>(p.x, q.i, n, xi);
        block_row_sums<C, G>(q.cnt, S, [&](int s, double* T) {
            const int j = pr.nb_b[q.base + s];
            double r[3] = {0.0, 0.0, 0.0};
            for (int d = 0; d < DIM; ++d) r[d] = xi[d] - p.x[(size_t)d * n + j];
            bdy_terms<DIM, SOIL>(c, p, t, j, r, pr.gw[q.base + s], T);
        });
    }
    const int row = blockIdx.x * ROWS + threadIdx.x;
    if (threadIdx.x >= ROWS || row >= count) return;
    const int i = list[row];
    double B[C];
    if (pr.cap_f && cnt[row] <= pr.cap_b) {
        for (int q = 0; q < C; ++q) B[q] = S[q][threadIdx.x];
    } else {
        double xi[3];
        load_x<DIM>(p.x, i, n, xi);
        for (int q = 0; q < C; ++q) B[q] = 0.0;
        for_neighbors<DIM>(c, p.x, t.pos32, cs, i, xi, true, [&](int j, const double* r, double rn) {
            if (!is_flow(p.mat_type[j])) return;
            double T[C];
            bdy_terms<DIM, SOIL>(c, p, t, j, r, kernel_W(c, rn), T);
            for (int q = 0; q < C; ++q) B[q] += T[q];
        });
    }
    const int ti = p.mat_type[i];
    const double f = t.CSPM_f[i], mV = p.m_V[i];
    const bool dyn = ti == MAT_RIGID && p.is_dynamic[i] != 0;
    double vt[3], rt;
    ld3(vt, p.v, n, i);
    for (int d = 0; d < 3; ++d) vt[d] = 2 * vt[d] - (d < DIM ? B[d < DIM ? d : 0] : 0.0) * f;
    st3(t.v_tmp, vt, n, i);
    if (!SOIL) {
        rt = c.rho0;
        const double pres = fmax(B[DIM] * f, 0.0);
        p.pressure[i] = pres;
        wc_record(c, pr.rec, i, vt, pres, rt, mV, false);
    } else {
        rt = c.solver == 2 ? fmax(B[DIM] * f, c.rho0) : c.rho0;
        double st[9];
        for (int q = 0; q < 9; ++q) {
            st[q] = B[(SOIL ? DIM + 1 : 0) + (SOIL ? q : 0)] * f;
            t.stress_tmp[(size_t)q * n + i] = st[q];
        }
        soil_record(c, pr.rec, i, vt, st, rt, mV);
    }
    t.density_tmp[i] = rt;
    // static rigid: rates stay zero; dynamic rigid: gravity, then the reaction.  Dummy and
    // repulsive particles have no rates: zero, as in the reference, where each particle's
    // never-written rates travel with it through the sort (the rate arrays here are not
    // reordered, so a slot may hold another particle's)
    t.d_density[i] = 0.0;
    for (int d = 0; d < 3; ++d) t.d_vel[(size_t)d * n + i] = dyn ? c.g[d] : 0.0;
}

// ---- repulsive particles (eng/solver_sph_base.py:675-689) ----
template <int DIM>
__device__ __forceinline__ void rep_force(const Consts& c, const double* r, double rn, double* acc) {
    double chi = (rn > 0.0 && rn < c.diam) ? 1.0 - rn / c.diam : 0.0;
    double gm = rn / c.h075;
    double f = 0.0;
    if (gm > 0 && gm <= 2.0 / 3.0) f = 2.0 / 3.0;
    else if (gm > 2.0 / 3.0 && gm <= 1) f = 2 * gm - 1.5 * (gm * gm);
    else if (gm > 1 && gm < 2) f = 0.5 * ((2 - gm) * (2 - gm));
    double s = c.rep_fac * chi * f / (rn * rn);
    for (int d = 0; d < DIM; ++d) acc[d] = acc[d] + s * r[d];
}

// One neighbour's term of calc_d_vel_task (eng/solver_sph_wc.py:34-71): viscosity
// (fluid, or boundary / rigid neighbours with the rho0 / rho~_i factor) plus pressure, for
// centre i and neighbour j of type tj; dvv = v~_i - v~_j, r = x_i - x_j, kd = grad W(r).
template <int DIM>
__device__ __forceinline__ void wc_force_pair(const Consts& c, int tj, double mVj, const double* dvv, double rti,
                                              double pri, double ptj, double rtj, const double* r, double rn,
                                              const double* kd, double* out) {
    const double mn = fmin(dotv<DIM>(dvv, r, PlainMul()), 0.0);
    const double den = rn * rn + c.eps_h2;
    double cv = 0.0;
    bool visc = false;
    if (tj == MAT_FLUID) { cv = c.visc_fac * mVj * mn / den; visc = true; }
    else if (tj == MAT_DUMMY || tj == MAT_REP || tj == MAT_RIGID) {
        cv = c.visc_fac * mVj * c.rho0 / rti * mn / den; visc = true;
    }
    const double cp = -c.rho0 * mVj * (pri + ptj / (rtj * rtj));
    for (int d = 0; d < DIM; ++d) {
        double pv = cp * kd[d];
        out[d] = visc ? cv * kd[d] + pv : 0.0 + pv;
    }
}

// The corrected gradient L_i grad W of a pair is the same in every loop of a step.  KC_MAKE
// forms it, KC_KEEP also stores it in the row, KC_READ reads it back (3D WCSPH: nine products and
// six additions of a pair for 24 bytes of stream; 118 k rows: 778 us with KC_KEEP, 578 with
// KC_READ).
enum { KC_MAKE = 0, KC_KEEP = 1, KC_READ = 2 };
template <int DIM>
__device__ __forceinline__ void corrected(const Consts& c, const double* L, const double* kd, double* kc) {
    if (c.corr == 1) matvec_corr<DIM>(L, kd, kc, PlainMul());
    else { kc[0] = kd[0]; kc[1] = kd[1]; kc[2] = kd[2]; }
}
// kd: grad W (KC_READ: not used); inside on_pipes.
template <int DIM, int KC, class M, class K>
__device__ __forceinline__ void row_gradient(const Consts& c, const Pairs64& pr, size_t slot, const double* L,
                                             bool L_ok, const double* kd, double* kc, M mul, K check) {
    if (KC == KC_READ) {
        for (int d = 0; d < DIM; ++d) kc[d] = pr.gc[d * pr.slots_f + slot];
    } else if (c.corr == 1) {
        check(L_ok);
        check.template all<DIM>(kd);
        matvec_corr<DIM>(L, kd, kc, mul);
    } else {
        for (int d = 0; d < DIM; ++d) kc[d] = kd[d];
    }
    check.template all<DIM>(kc);
}
template <int DIM, int KC>
__device__ __forceinline__ void load_gradient(const Pairs64& pr, size_t slot, double* kd) {
    if (KC != KC_READ)
        for (int d = 0; d < DIM; ++d) kd[d] = pr.gk[d * pr.slots_f + slot];
}
template <int DIM, int KC>
__device__ __forceinline__ void keep_gradient(const Pairs64& pr, size_t slot, const double* kc) {
    if (KC == KC_KEEP)
        for (int d = 0; d < DIM; ++d) pr.gc[d * pr.slots_f + slot] = kc[d];
}

// One neighbour's WCSPH terms: continuity, then the acceleration (DIM), from the neighbour's
// record (v~, P = p / rho~^2, m_V, viscosity factor, -rho0 m_V) and the pair geometry
// (den.y: den.x's divisor() bits).
struct Divisor {  // a divisor with its divisor() bits
    double b;
    unsigned long long X;
    __device__ __forceinline__ explicit Divisor(double v) : b(v), X(divisor(v)) {}
};
template <int DIM, class M, class Q, class K>
__device__ __forceinline__ void wc_terms(bool fluid, const double* v, double P, double mV, double cvj, double cC,
                                         const double* vti, const Divisor& rti, double pri, const double* r,
                                         double2 den, const double* kd, const double* kc, double* T, M mul, Q quot,
                                         K check) {
    double dvv[3], a[3];
    for (int d = 0; d < DIM; ++d) dvv[d] = vti[d] - v[d];
    check(mV);
    check.template all<DIM>(dvv);
    check.template all<DIM>(r);
    for (int d = 0; d < DIM; ++d) a[d] = mul(mV, dvv[d]);
    T[0] = dotv<DIM>(a, kc, mul);
    const double mn = min0(dotv<DIM>(dvv, r, mul));
    double cv = cvj, cp = pri + P;
    check(cv);
    check(cp);
    check(cC);
    check(mn);
    if (!fluid) {
        check(rti.X != 0ull);
        cv = quot(cv, rti.b, rti.X);
    }
    const unsigned long long X = (unsigned long long)__double_as_longlong(den.y);
    check(X != 0ull);
    cv = quot(mul(cv, mn), den.x, X);
    cp = mul(cC, cp);
    check.template all<DIM>(kd);
    for (int d = 0; d < DIM; ++d) T[1 + d] = cv * kd[d] + mul(cp, kd[d]);  // one product on each pipe
}

// ---- WCSPH rates (eng/solver_sph_wc.py:108-126) ----
template <int DIM, int G, int KC>
__global__ void __launch_bounds__(ROWS * G, G == 8 ? 2 : DIM == 3 && KC == KC_READ ? 6 : 5) k_wc_rates(Consts c, Persist64 p, Trans64 t, const int* __restrict__ cs,
                                                       const int* __restrict__ list, int count, Pairs64 pr) {
    constexpr int C = 1 + DIM;
    __shared__ double S[C][ROWS];
    const int n = c.n;
    if (pr.cap_f) {
        const RowRef q = row_ref<G>(list, count, pr.cnt, pr.cap_f);
        double xi[3], vti[3], L[9];
        load_x<DIM>(p.x, q.i, n, xi);
        for (int d = 0; d < 3; ++d) vti[d] = t.v_tmp[(size_t)d * n + q.i];
        const Divisor rti(t.density_tmp[q.i]);
        const double pri = pr.rec[(size_t)8 * q.i + 3];
        if (c.corr == 1 && KC != KC_READ)
            for (int e = 0; e < 9; ++e) L[e] = t.CSPM_L[(size_t)e * n + q.i];
        const bool L_ok = c.corr == 1 && KC != KC_READ && usable_m<DIM>(L);
        block_row_sums<C, G>(q.cnt, S, [&](int s, double* T) {
            const size_t slot = q.base + s;
            const int ent = pr.nb_f[slot], j = nb_index(ent);
            const double2* rj = reinterpret_cast<const double2*>(pr.rec + (size_t)8 * j);
            const double2 r0 = rj[0], r1 = rj[1], r2 = rj[2], r3 = rj[3];
            const double2 den = pr.gden[slot];
            double r[3] = {0.0, 0.0, 0.0}, kd[3] = {0.0, 0.0, 0.0}, kc[3];
            for (int d = 0; d < DIM; ++d) {
                r[d] = xi[d] - p.x[(size_t)d * n + j];
                kd[d] = pr.gk[d * pr.slots_f + slot];
            }
            const double v[3] = {r0.x, r0.y, r1.x};
            on_pipes([&](auto mul, auto quot, auto check) {
                row_gradient<DIM, KC>(c, pr, slot, L, L_ok, kd, kc, mul, check);
                wc_terms<DIM>(nb_flow(ent), v, r1.y, r2.x, r2.y, r3.x, vti, rti, pri, r, den, kd, kc, T, mul, quot, check);
            });
            keep_gradient<DIM, KC>(pr, slot, kc);
        });
    }
    const int row = blockIdx.x * ROWS + threadIdx.x;
    if (threadIdx.x >= ROWS || row >= count) return;
    const int i = list[row];
    const Divisor rti(t.density_tmp[i]);
    double A[C];
    const bool listed = pr.cap_f && pr.cnt[row] <= pr.cap_f;
    const bool rep = c.boundary == 3 || c.boundary == 4;
    double xi[3];
    load_x<DIM>(p.x, i, n, xi);
    if (listed) {
        for (int q = 0; q < C; ++q) A[q] = S[q][threadIdx.x];
    } else {
        double vti[3], L[9];
        for (int d = 0; d < 3; ++d) vti[d] = t.v_tmp[(size_t)d * n + i];
        const double pri = pr.rec[(size_t)8 * i + 3];
        if (c.corr == 1)
            for (int q = 0; q < 9; ++q) L[q] = t.CSPM_L[(size_t)q * n + i];
        for (int q = 0; q < C; ++q) A[q] = 0.0;
        for_neighbors<DIM>(c, p.x, t.pos32, cs, i, xi, true, [&](int j, const double* r, double rn) {
            const double* rj = pr.rec + (size_t)8 * j;
            double kd[3], kc[3], T[C];
            kernel_dW<DIM>(c, r, rn, kd);
            corrected<DIM>(c, L, kd, kc);
            const double den = rn * rn + c.eps_h2;
            wc_terms<DIM>(p.mat_type[j] == MAT_FLUID, rj, rj[3], rj[4], rj[5], rj[6], vti, rti, pri, r,
                          make_double2(den, 0.0), kd, kc, T, SlowMul(), SlowQuot(), NoCheck());
            for (int q = 0; q < C; ++q) A[q] += T[q];
        });
    }
    if (rep) {  // a separate walk: the reference adds these after the whole acceleration sum
        for_neighbors<DIM>(c, p.x, t.pos32, cs, i, xi, true, [&](int j, const double* r, double rn) {
            if (p.mat_type[j] == MAT_REP) rep_force<DIM>(c, r, rn, A + 1);
        });
    }
    t.d_density[i] = A[0] * rti.b;
    for (int d = 0; d < DIM; ++d) t.d_vel[(size_t)d * n + i] = A[1 + d] + c.g[d];
    if (DIM == 2) t.d_vel[2 * (size_t)n + i] = 0.0 + c.g[2];
}

// ---- soil helpers ----
__device__ __forceinline__ void damping_acc(const Consts& c, double rti, const double* vti, double* out, int dim) {
    double s = -c.damp_eps * sqrt(c.damp_E / (rti * c.h2));
    for (int d = 0; d < dim; ++d) out[d] = s * vti[d];
}

// One neighbour's velocity-gradient terms (DIM x DIM) and continuity term (last): the
// continuity product m_V (v_i - v_j) is the exact negation of the gradient's, so its dot
// product is the negated trace.
template <int DIM, class M, class K>
__device__ __forceinline__ void vgrad_terms(const double* v, double mV, const double* vti, const double* kc, double* T,
                                            M mul, K check) {
    double dv[3];
    for (int a = 0; a < DIM; ++a) dv[a] = v[a] - vti[a];
    check(mV);
    check.template all<DIM>(dv);
    for (int a = 0; a < DIM; ++a) {
        const double av = mul(mV, dv[a]);
        for (int b = 0; b < DIM; ++b) T[a * DIM + b] = mul(av, kc[b]);
    }
    double s = T[0] + T[DIM + 1];
    if (DIM == 3) s = s + T[8];
    T[DIM * DIM] = -s;
}

// mu(I) loop 1 (eng/solver_sph_muI.py:67-92): velocity gradient, continuity, pressure from
// density (not density_tmp), mu(I) stress, equivalent strain rate.
template <int DIM, int G, int KC>
__global__ void __launch_bounds__(ROWS * G) k_mui_stress(Consts c, Persist64 p, Trans64 t, const int* __restrict__ cs,
                                                         const int* __restrict__ list, int count, Pairs64 pr) {
    constexpr int C = DIM * DIM + 1;
    __shared__ double S[C][ROWS];
    const int n = c.n;
    if (pr.cap_f) {
        const RowRef q = row_ref<G>(list, count, pr.cnt, pr.cap_f);
        double vti[3], L[9];
        for (int d = 0; d < 3; ++d) vti[d] = t.v_tmp[(size_t)d * n + q.i];
        if (c.corr == 1 && KC != KC_READ)
            for (int e = 0; e < 9; ++e) L[e] = t.CSPM_L[(size_t)e * n + q.i];
        const bool L_ok = c.corr == 1 && KC != KC_READ && usable_m<DIM>(L);
        block_row_sums<C, G>(q.cnt, S, [&](int s, double* T) {
            const size_t slot = q.base + s;
            const int j = nb_index(pr.nb_f[slot]);
            double kd[3], kc[3], v[3];
            for (int d = 0; d < DIM; ++d) v[d] = t.v_tmp[(size_t)d * n + j];
            load_gradient<DIM, KC>(pr, slot, kd);
            const double mVj = p.m_V[j];
            on_pipes([&](auto mul, auto, auto check) {
                row_gradient<DIM, KC>(c, pr, slot, L, L_ok, kd, kc, mul, check);
                vgrad_terms<DIM>(v, mVj, vti, kc, T, mul, check);
            });
            keep_gradient<DIM, KC>(pr, slot, kc);
        });
    }
    const int row = blockIdx.x * ROWS + threadIdx.x;
    if (threadIdx.x >= ROWS || row >= count) return;
    const int i = list[row];
    double A[C], vti[3];
    for (int d = 0; d < 3; ++d) vti[d] = t.v_tmp[(size_t)d * n + i];
    if (pr.cap_f && pr.cnt[row] <= pr.cap_f) {
        for (int q = 0; q < C; ++q) A[q] = S[q][threadIdx.x];
    } else {
        double xi[3], L[9];
        load_x<DIM>(p.x, i, n, xi);
        if (c.corr == 1)
            for (int q = 0; q < 9; ++q) L[q] = t.CSPM_L[(size_t)q * n + i];
        for (int q = 0; q < C; ++q) A[q] = 0.0;
        for_neighbors<DIM>(c, p.x, t.pos32, cs, i, xi, true, [&](int j, const double* r, double rn) {
            double kd[3], kc[3], v[3], T[C];
            kernel_dW<DIM>(c, r, rn, kd);
            corrected<DIM>(c, L, kd, kc);
            for (int d = 0; d < DIM; ++d) v[d] = t.v_tmp[(size_t)d * n + j];
            vgrad_terms<DIM>(v, p.m_V[j], vti, kc, T, SlowMul(), NoCheck());
            for (int q = 0; q < C; ++q) A[q] += T[q];
        });
    }
    double vg[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (int a = 0; a < DIM; ++a)
        for (int b = 0; b < DIM; ++b) vg[3 * a + b] = A[a * DIM + b];
    const double rti = t.density_tmp[i];
    for (int q = 0; q < 9; ++q) t.v_grad[(size_t)q * n + i] = vg[q];
    t.d_density[i] = A[DIM * DIM] * rti;
    const double pr_i = fmax(c.vsound2 * (p.density[i] - c.rho0), 0.0);
    p.pressure[i] = pr_i;
    double er[9], st[9];
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) er[3 * a + b] = 0.5 * (vg[3 * a + b] + vg[3 * b + a]);
    const double dbdot = sqrt(0.5 * msum_sq(er)) + EPS;
    const double sc = 0.0 + (c.coh + pr_i * c.mu) / dbdot;
    for (int q = 0; q < 9; ++q) {
        st[q] = sc * er[q] - pr_i * ((q % 4 == 0) ? 1.0 : 0.0);
        t.stress_tmp[(size_t)q * n + i] = st[q];
    }
    const double t3 = mtrace(er) / 3.0;
    double ed[9];
    for (int q = 0; q < 9; ++q) ed[q] = er[q] - t3 * ((q % 4 == 0) ? 1.0 : 0.0);
    t.d_strain_equ[i] = sqrt(msum_sq(ed) * 2 / 3);
    soil_record(c, pr.rec, i, vti, st, rti, p.m_V[i]);
}

// Stress-divergence sum (eng/solver_sph_muI.py:39-46), shared by mu(I) and DP.
template <int DIM>
__device__ __forceinline__ void stress_div_val(const double* sti, double ri2, const double* stj, double rtj,
                                               double mVj, const double* kc, double* out) {
    const double rj2 = rtj * rtj;
    const double sc = mVj * rtj;
    for (int a = 0; a < DIM; ++a) {
        double s = 0.0;
        for (int b = 0; b < DIM; ++b) {
            double m = stj[3 * a + b] / rj2 + sti[3 * a + b] / ri2;
            double v = (sc * m) * kc[b];
            s = b == 0 ? v : s + v;
        }
        out[a] = s;
    }
}
// The same sum from the neighbour's record: S_j = stress_j / rho~_j^2 (DIM x DIM), sc = m_V rho~_j,
// and S_i likewise.
template <int DIM, class M, class K>
__device__ __forceinline__ void stress_div_rec(const double* Si, const double* Sj, double sc, const double* kc,
                                               double* out, M mul, K check) {
    double m[DIM * DIM];
    for (int q = 0; q < DIM * DIM; ++q) m[q] = Sj[q] + Si[q];
    check(sc);
    check.template all<DIM * DIM>(m);
    for (int q = 0; q < DIM * DIM; ++q) m[q] = mul(mul(sc, m[q]), kc[q % DIM]);
    for (int a = 0; a < DIM; ++a) {
        out[a] = m[a * DIM] + m[a * DIM + 1];
        if (DIM == 3) out[a] = out[a] + m[a * DIM + 2];
    }
}

// A soil record: v~ (DIM), m_V, m_V rho~, stress~ / rho~^2 (DIM x DIM).
template <int DIM>
struct SoilRec {
    double a[DIM == 2 ? 8 : 16];
    __device__ __forceinline__ SoilRec(const double* rec, int j) {
        constexpr int N = DIM == 2 ? 8 : 16;
        const double2* q = reinterpret_cast<const double2*>(rec + (size_t)N * j);
#pragma unroll
        for (int e = 0; e < N / 2 - (DIM == 3 ? 1 : 0); ++e) {
            const double2 w = q[e];
            a[2 * e] = w.x;
            a[2 * e + 1] = w.y;
        }
    }
    __device__ __forceinline__ const double* v() const { return a; }
    __device__ __forceinline__ double mV() const { return a[DIM]; }
    __device__ __forceinline__ double sc() const { return a[DIM + 1]; }
    __device__ __forceinline__ const double* S() const { return a + DIM + 2; }
};

// mu(I) loop 2 (eng/solver_sph_muI.py:113-128) and the whole Drucker-Prager loop
// (eng/solver_sph_dp.py:236-270): stress divergence, and for Drucker-Prager the velocity
// gradient and continuity in the same walk.  Component order: acceleration, gradient, continuity.
template <int DIM, int G, bool DP, int KC>
__device__ __forceinline__ void soil_sums(const Consts& c, const Persist64& p, const Trans64& t,
                                          const int* __restrict__ cs, const int* __restrict__ list, int count,
                                          const Pairs64& pr, double (*S)[ROWS], double* A) {
    constexpr int C = DIM + (DP ? DIM * DIM + 1 : 0);
    const int n = c.n;
    if (pr.cap_f) {
        const RowRef q = row_ref<G>(list, count, pr.cnt, pr.cap_f);
        double L[9];
        if (c.corr == 1 && KC != KC_READ)
            for (int e = 0; e < 9; ++e) L[e] = t.CSPM_L[(size_t)e * n + q.i];
        const bool L_ok = c.corr == 1 && KC != KC_READ && usable_m<DIM>(L);
        const SoilRec<DIM> ri(pr.rec, q.i);
        block_row_sums<C, G>(q.cnt, S, [&](int s, double* T) {
            const size_t slot = q.base + s;
            const int j = nb_index(pr.nb_f[slot]);
            double kd[3], kc[3];
            load_gradient<DIM, KC>(pr, slot, kd);
            const SoilRec<DIM> rj(pr.rec, j);
            on_pipes([&](auto mul, auto, auto check) {
                row_gradient<DIM, KC>(c, pr, slot, L, L_ok, kd, kc, mul, check);
                stress_div_rec<DIM>(ri.S(), rj.S(), rj.sc(), kc, T, mul, check);
                if (DP) vgrad_terms<DIM>(rj.v(), rj.mV(), ri.v(), kc, T + DIM, mul, check);
            });
            keep_gradient<DIM, KC>(pr, slot, kc);
        });
    }
    const int row = blockIdx.x * ROWS + threadIdx.x;
    if (threadIdx.x >= ROWS || row >= count) return;
    const int i = list[row];
    const bool rep = c.boundary == 3 || c.boundary == 4;
    double xi[3];
    load_x<DIM>(p.x, i, n, xi);
    if (pr.cap_f && pr.cnt[row] <= pr.cap_f) {
        for (int q = 0; q < C; ++q) A[q] = S[q][threadIdx.x];
    } else {
        double L[9];
        if (c.corr == 1)
            for (int q = 0; q < 9; ++q) L[q] = t.CSPM_L[(size_t)q * n + i];
        const SoilRec<DIM> ri(pr.rec, i);
        for (int q = 0; q < C; ++q) A[q] = 0.0;
        for_neighbors<DIM>(c, p.x, t.pos32, cs, i, xi, true, [&](int j, const double* r, double rn) {
            double kd[3], kc[3], T[C];
            kernel_dW<DIM>(c, r, rn, kd);
            corrected<DIM>(c, L, kd, kc);
            const SoilRec<DIM> rj(pr.rec, j);
            stress_div_rec<DIM>(ri.S(), rj.S(), rj.sc(), kc, T, SlowMul(), NoCheck());
            if (DP) vgrad_terms<DIM>(rj.v(), rj.mV(), ri.v(), kc, T + DIM, SlowMul(), NoCheck());
            for (int q = 0; q < C; ++q) A[q] += T[q];
        });
    }
    // repulsive forces (mu(I) only: the Drucker-Prager loop of the reference adds none)
    if (rep && !DP)
        for_neighbors<DIM>(c, p.x, t.pos32, cs, i, xi, true, [&](int j, const double* r, double rn) {
            if (p.mat_type[j] == MAT_REP) rep_force<DIM>(c, r, rn, A);
        });
}

template <int DIM, int G, int KC>
__global__ void __launch_bounds__(ROWS * G) k_mui_mom(Consts c, Persist64 p, Trans64 t, const int* __restrict__ cs,
                                                      const int* __restrict__ list, int count, Pairs64 pr) {
    __shared__ double S[DIM][ROWS];
    double dv[3] = {0, 0, 0};
    soil_sums<DIM, G, false, KC>(c, p, t, cs, list, count, pr, S, dv);
    const int row = blockIdx.x * ROWS + threadIdx.x;
    if (threadIdx.x >= ROWS || row >= count) return;
    const int i = list[row];
    const int n = c.n;
    double vti[3], fd[3] = {0, 0, 0};
    for (int d = 0; d < 3; ++d) vti[d] = t.v_tmp[(size_t)d * n + i];
    damping_acc(c, t.density_tmp[i], vti, fd, 3);
    for (int d = 0; d < 3; ++d) t.d_vel[(size_t)d * n + i] = (dv[d] + c.g[d]) + fd[d];
}

// ---- DP rates (eng/solver_sph_dp.py:236-270, Bui 2008 :172-208) ----
// The 2D bound holds five blocks of 128 threads on an SM: 20,000 rows then run in one wave
// (8 lanes and no bound: two waves and a nearly empty third, 2,975 us per ten steps; 2,447 now).
template <int DIM, int G, int KC>
__global__ void __launch_bounds__(ROWS * G, DIM == 2 ? 20 / G : 1) k_dp_rates(Consts c, Persist64 p, Trans64 t, const int* __restrict__ cs,
                                                       const int* __restrict__ list, int count, Pairs64 pr) {
    constexpr int C = DIM + DIM * DIM + 1;
    __shared__ double S[C][ROWS];
    double A[C];
    soil_sums<DIM, G, true, KC>(c, p, t, cs, list, count, pr, S, A);
    const int row = blockIdx.x * ROWS + threadIdx.x;
    if (threadIdx.x >= ROWS || row >= count) return;
    const int i = list[row];
    const int n = c.n;
    double vti[3], sti[9], dv[3] = {0, 0, 0};
    for (int d = 0; d < 3; ++d) vti[d] = t.v_tmp[(size_t)d * n + i];
    for (int q = 0; q < 9; ++q) sti[q] = t.stress_tmp[(size_t)q * n + i];
    const double rti = t.density_tmp[i];
    double vg[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (int a = 0; a < DIM; ++a) {
        dv[a] = A[a];
        for (int b = 0; b < DIM; ++b) vg[3 * a + b] = A[DIM + a * DIM + b];
    }
    const double dd = A[C - 1];
    for (int q = 0; q < 9; ++q) t.v_grad[(size_t)q * n + i] = vg[q];
    t.d_density[i] = dd * rti;
    // Bui 2008 stress rate
    double s[9], I1, sJ2, f_old;
    dp_inv(c, sti, s, I1, sJ2, f_old);
    double er[9], wr[9];
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) {
            er[3 * a + b] = 0.5 * (vg[3 * a + b] + vg[3 * b + a]);
            wr[3 * a + b] = 0.5 * (vg[3 * a + b] - vg[3 * b + a]);
        }
    double J[9];
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b)
            J[3 * a + b] = sti[3 * a] * wr[3 * b] + sti[3 * a + 1] * wr[3 * b + 1] + sti[3 * a + 2] * wr[3 * b + 2]
                         + sti[b] * wr[3 * a] + sti[3 + b] * wr[3 * a + 1] + sti[6 + b] * wr[3 * a + 2];
    const double tr = mtrace(er);
    double ed[9], te[9];
    for (int q = 0; q < 9; ++q) {
        ed[q] = er[q] - (tr / 3.0) * ((q % 4 == 0) ? 1.0 : 0.0);
        te[q] = c.twoG * ed[q] + (c.Km * tr) * ((q % 4 == 0) ? 1.0 : 0.0);
    }
    const bool plastic = f_old >= -EPS_F && sJ2 > EPS;
    double lam = 0.0;
    double ds[9];
    for (int q = 0; q < 9; ++q) {
        double tg = 0.0;
        if (plastic && q == 0) lam = (c.three_aK * tr + (c.Gm / sJ2) * msum_prod(s, er)) / c.lam_den;
        if (plastic) tg = lam * (c.nine_K_sin * ((q % 4 == 0) ? 1.0 : 0.0) + c.Gm / sJ2 * s[q]);
        ds[q] = (J[q] + te[q]) - tg;
    }
    for (int q = 0; q < 9; ++q) t.d_stress[(size_t)q * n + i] = ds[q];
    t.d_strain_equ[i] = sqrt(msum_sq(ed) * 2 / 3);
    double dep = 0.0;
    if (plastic) {
        const double gp = sJ2 + 3 * I1 * c.sin_dila;
        const double gd = gp - 0.0;  // g_p is never written by the reference (eng/particle_func.py:52)
        double ep[9];
        for (int q = 0; q < 9; ++q) {
            double v = fabs(ds[q]) > EPS ? gd / ds[q] : 0.0;
            ep[q] = lam * v;
        }
        const double t3 = mtrace(ep) / 3.0;
        double epd[9];
        for (int q = 0; q < 9; ++q) epd[q] = ep[q] - t3 * ((q % 4 == 0) ? 1.0 : 0.0);
        dep = sqrt(msum_sq(epd) * 2 / 3);
    }
    t.d_strain_equ_p[i] = dep;
    double fd[3] = {0, 0, 0};
    damping_acc(c, rti, vti, fd, 3);
    for (int d = 0; d < 3; ++d) t.d_vel[(size_t)d * n + i] = (dv[d] + c.g[d]) + fd[d];
}

// ---- advect_pos with XSPH (eng/solver_sph_base.py:224-238), two phases ----
template <int DIM, int G>
__global__ void __launch_bounds__(ROWS * G) k_xsph(Consts c, Persist64 p, Trans64 t, const int* __restrict__ cs,
                                                   const int* __restrict__ list, int count, Pairs64 pr) {
    __shared__ double S[DIM][ROWS];
    const int n = c.n;
    const int tf = c.flow_type;
    if (pr.cap_f) {
        const RowRef q = row_ref<G>(list, count, pr.cnt, pr.cap_f);
        double xi[3], vi[3];
        load_x<DIM>(p.x, q.i, n, xi);
        for (int d = 0; d < 3; ++d) vi[d] = p.v[(size_t)d * n + q.i];
        block_row_sums<DIM, G>(q.cnt, S, [&](int s, double* T) {
            const int ent = pr.nb_f[q.base + s];
            if (!nb_flow(ent)) return;
            const double w = pair_W<DIM>(c, p.x, xi, ent);
            const double mVj = p.m_V[ent];
            double dv[3];
            for (int d = 0; d < DIM; ++d) dv[d] = p.v[(size_t)d * n + ent] - vi[d];
            on_pipe(usable(mVj) && usable(w) && usable_v<DIM>(dv), [&](auto mul) {
                for (int d = 0; d < DIM; ++d) T[d] = mul(mul(mVj, dv[d]), w);
            });
        });
    }
    const int row = blockIdx.x * ROWS + threadIdx.x;
    if (threadIdx.x >= ROWS || row >= count) return;
    const int i = list[row];
    if (!p.is_dynamic[i]) return;
    double s[3] = {0, 0, 0};
    if (pr.cap_f && pr.cnt[row] <= pr.cap_f) {
        for (int d = 0; d < DIM; ++d) s[d] = S[d][threadIdx.x];
    } else {
        double xi[3], vi[3];
        load_x<DIM>(p.x, i, n, xi);
        for (int d = 0; d < 3; ++d) vi[d] = p.v[(size_t)d * n + i];
        for_neighbors<DIM>(c, p.x, t.pos32, cs, i, xi, true, [&](int j, const double* r, double rn) {
            if (p.mat_type[j] != tf) return;
            const double w = kernel_W(c, rn);
            const double mVj = p.m_V[j];
            for (int d = 0; d < DIM; ++d) s[d] += mVj * (p.v[(size_t)d * n + j] - vi[d]) * w;
        });
    }
    for (int d = 0; d < 3; ++d) t.aux3[(size_t)d * n + i] = s[d];
}

// Dynamic rigid particles move by the XSPH sum over their own kind (rigid rows list flow
// neighbours only, so these walk the cells).
template <int DIM>
__global__ void k_xsph_rigid(Consts c, Persist64 p, Trans64 t, const int* __restrict__ cs,
                             const int* __restrict__ list, int count) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= count) return;
    const int i = list[k];
    const int n = c.n;
    const int ti = p.mat_type[i];
    if (!(ti > 0 && p.is_dynamic[i])) return;
    double xi[3], vi[3];
    load_x<DIM>(p.x, i, n, xi);
    for (int d = 0; d < 3; ++d) vi[d] = p.v[(size_t)d * n + i];
    double s[3] = {0, 0, 0};
    for_neighbors<DIM>(c, p.x, t.pos32, cs, i, xi, true, [&](int j, const double* r, double rn) {
        if (p.mat_type[j] != ti) return;
        const double w = kernel_W(c, rn);
        const double mVj = p.m_V[j];
        for (int d = 0; d < DIM; ++d) s[d] += mVj * (p.v[(size_t)d * n + j] - vi[d]) * w;
    });
    for (int d = 0; d < 3; ++d) t.aux3[(size_t)d * n + i] = s[d];
}

// Stress regularisation after advect_pos: centres use their moved positions, candidate
// cells come from this step's sort (eng/solver_sph_muI.py:151-156).  The rows are rebuilt from
// the moved positions first (flow neighbours only).  The loop's stress is stress_tmp, which the
// reference copies into stress just before (:148), so the sums read it there and go straight
// into stress.  In 2D the four out-of-plane shears are zero unless a caller wrote some: their
// products (+-0, which no sum starting at +0 notices) are formed only where one is not.
template <int DIM, int G>
__global__ void __launch_bounds__(ROWS * G) k_post_mui(Consts c, Persist64 p, Trans64 t, const int* __restrict__ cs,
                                                       const int* __restrict__ list, int count, Pairs64 pr) {
    constexpr int C = 9;
    __shared__ double S[C][ROWS];
    const int n = c.n;
    if (pr.cap_f) {
        const RowRef q = row_ref<G>(list, count, pr.cnt, pr.cap_f);
        double xi[3];
        load_x<DIM>(p.x, q.i, n, xi);
        block_row_sums<C, G>(q.cnt, S, [&](int s, double* T) {
            const int j = pr.nb_f[q.base + s];
            const double w = pair_W<DIM>(c, p.x, xi, j);
            const double mVj = p.m_V[j];
            double st[9];
            ld9(st, t.stress_tmp, n, j);
            const bool ok = usable(mVj) && usable(w);
            const bool plane = usable(st[0]) && usable(st[1]) && usable(st[3]) && usable(st[4]) && usable(st[8]);
            on_pipe(ok && plane, [&](auto mul) {
                T[0] = mul(mul(mVj, st[0]), w);
                T[1] = mul(mul(mVj, st[1]), w);
                T[3] = mul(mul(mVj, st[3]), w);
                T[4] = mul(mul(mVj, st[4]), w);
                T[8] = mul(mul(mVj, st[8]), w);
            });
            // (a factor that is not finite makes them NaN, not zero)
            if (DIM == 3 || !ok || !(zero(st[2]) && zero(st[5]) && zero(st[6]) && zero(st[7]))) {
                on_pipe(ok && usable(st[2]) && usable(st[5]) && usable(st[6]) && usable(st[7]), [&](auto mul) {
                    T[2] = mul(mul(mVj, st[2]), w);
                    T[5] = mul(mul(mVj, st[5]), w);
                    T[6] = mul(mul(mVj, st[6]), w);
                    T[7] = mul(mul(mVj, st[7]), w);
                });
            }
        });
    }
    const int row = blockIdx.x * ROWS + threadIdx.x;
    if (threadIdx.x >= ROWS || row >= count) return;
    const int i = list[row];
    double s[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    if (pr.cap_f && pr.cnt[row] <= pr.cap_f) {
        for (int q = 0; q < 9; ++q) s[q] = S[q][threadIdx.x];
    } else {
        double xi[3];
        load_x<DIM>(p.x, i, n, xi);
        for_neighbors<DIM>(c, p.x, t.pos32, cs, i, xi, false, [&](int j, const double* r, double rn) {
            if (p.mat_type[j] != MAT_SOIL) return;
            const double w = kernel_W(c, rn);
            const double mVj = p.m_V[j];
            for (int q = 0; q < 9; ++q) s[q] += mVj * t.stress_tmp[(size_t)q * n + j] * w;
        });
    }
    const double f = t.CSPM_f[i];
    for (int q = 0; q < 9; ++q) s[q] = s[q] * f;
    st9(p.stress, s, n, i);
}

// ---- per-particle passes ----
// The passes of a step between its pair loops, in the order of the bits; every value they
// exchange belongs to one particle, so a launch runs all that lie between two loops (a leap-frog
// step: 3 launches instead of 7 of about 3 us each on a small scene).
enum : unsigned {
    OP_INIT = 1, OP_RK_INIT = 2, OP_RK_UPDATE = 4, OP_HALF = 8, OP_RK_STAGE = 16, OP_FULL = 32, OP_RK_FINAL = 64,
    OP_PRE = 128, OP_POS = 256, OP_POST = 512
};
// All loads come first and all stores last: interleaved, each store held back the next plane's
// load (the compiler cannot tell the planes apart) and the pass was a chain of round trips.
template <bool SOIL>
__global__ void __launch_bounds__(TPB) k_particle(Consts c, Persist64 p, Trans64 t, Pairs64 pr, unsigned ops, int m,
                                                  int* err) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    const int ti = p.mat_type[i];
    if (ti <= 0) return;
    const size_t n = c.n;
    const bool soil = SOIL && ti == MAT_SOIL, dp = soil && c.solver == 3;
    const bool pre = (ops & OP_PRE) && ti == c.flow_type;
    const bool post = (ops & OP_POST) && ti == (SOIL ? MAT_SOIL : MAT_FLUID);
    const bool has = ops & (OP_INIT | OP_RK_STAGE);  // rho~, v~ set here
    double rho = 0, mass = 0, mV = 0, rt = 0, dd = 0, ad = 0, v[3], x[3], vt[3], dv[3], av[3];
    double st[9], stt[9], ds[9], as[9], eq = 0, eqp = 0, deq = 0, deqp = 0, xs[3] = {0, 0, 0};
    const unsigned rates_in = OP_RK_UPDATE | OP_HALF | OP_RK_STAGE | OP_FULL;
    const bool upd_rho = ops & (OP_FULL | OP_RK_FINAL);
    if ((ops & (OP_INIT | OP_RK_STAGE)) || upd_rho || post) rho = p.density[i];
    if (ops & (OP_INIT | OP_RK_STAGE | OP_FULL | OP_RK_FINAL | OP_POS)) ld3(v, p.v, n, i);
    if (ops & (OP_HALF | OP_RK_STAGE | OP_FULL | OP_RK_FINAL) || post) mass = p.mass[i];
    if (ops & rates_in) { dd = t.d_density[i]; ld3(dv, t.d_vel, n, i); }
    if ((ops & (OP_RK_UPDATE | OP_RK_FINAL)) && !(ops & OP_RK_INIT)) { ad = t.d_density_RK[i]; ld3(av, t.d_vel_RK, n, i); }
    if ((ops & OP_HALF) || (pre && !has)) { rt = t.density_tmp[i]; ld3(vt, t.v_tmp, n, i); }
    if (pre && !(ops & (OP_HALF | OP_RK_STAGE))) mV = p.m_V[i];
    const bool xsph = (ops & OP_POS) && c.xsph && p.is_dynamic[i];
    if (ops & OP_POS) {
        ld3(x, p.x, n, i);
        if (xsph) ld3(xs, t.aux3, n, i);
    }
    if (SOIL && soil) {
        if ((ops & OP_INIT) || (dp && ((ops & (OP_RK_STAGE | OP_FULL | OP_RK_FINAL)) || post))) ld9(st, p.stress, n, i);
        if (dp && ((ops & OP_HALF) || (pre && !has))) ld9(stt, t.stress_tmp, n, i);
        if (dp && (ops & rates_in)) ld9(ds, t.d_stress, n, i);
        if (dp && (ops & (OP_RK_UPDATE | OP_RK_FINAL)) && !(ops & OP_RK_INIT)) ld9(as, t.d_stress_RK, n, i);
        if (post) {
            eq = p.strain_equ[i];
            deq = t.d_strain_equ[i];
            if (dp) { eqp = p.strain_equ_p[i]; deqp = t.d_strain_equ_p[i]; }
        }
    }

    // init_real2tmp (eng/solver_sph_base.py:67-74)
    if (ops & OP_INIT) {
        rt = rho;
        for (int d = 0; d < 3; ++d) vt[d] = v[d];
        if (SOIL && soil)
            for (int q = 0; q < 9; ++q) stt[q] = st[q];
    }
    // the integrators (eng/solver_sph_base.py:79-170)
    if (ops & OP_RK_INIT) {
        ad = 0.0;
        for (int d = 0; d < 3; ++d) av[d] = 0.0;
        if (SOIL && dp)
            for (int q = 0; q < 9; ++q) as[q] = 0.0;
    }
    if (ops & OP_RK_UPDATE) {
        ad += dd * m;
        for (int d = 0; d < 3; ++d) av[d] += dv[d] * m;
        if (SOIL && dp)
            for (int q = 0; q < 9; ++q) as[q] += (double)m * ds[q];
    }
    if (ops & OP_HALF) {
        rt = rt + c.hdt * dd;
        mV = mass / rt;
        for (int d = 0; d < 3; ++d) vt[d] += c.hdt * dv[d];
        if (SOIL && dp)
            for (int q = 0; q < 9; ++q) stt[q] += c.hdt * ds[q];
    }
    if (ops & OP_RK_STAGE) {
        rt = c.hdt * dd + rho;
        mV = mass / rt;
        for (int d = 0; d < 3; ++d) vt[d] = c.hdt * dv[d] + v[d];
        if (SOIL && dp)
            for (int q = 0; q < 9; ++q) stt[q] = c.hdt * ds[q] + st[q];
    }
    bool bad = false;
    if (ops & OP_FULL) {
        rho = rho + c.dt * dd;
        mV = mass / rho;
        for (int d = 0; d < 3; ++d) v[d] += c.dt * dv[d];
        bad = !isfinite(rho);
        if (SOIL && dp)
            for (int q = 0; q < 9; ++q) st[q] += c.dt * ds[q];
    }
    if (ops & OP_RK_FINAL) {
        rho = rho + c.dt6 * ad;
        mV = mass / rho;
        for (int d = 0; d < 3; ++d) v[d] += c.dt6 * av[d];
        bad = !isfinite(rho);
        if (SOIL && dp)
            for (int q = 0; q < 9; ++q) st[q] += c.dt6 * as[q];
    }
    // first phase of one_step: Tait EOS (eng/solver_sph_wc.py:86-88) or stress adaptation
    // (eng/solver_sph_dp.py:215-217), and the record the loops read
    double pres = 0.0;
    if (pre) {
        if (!SOIL) {
            const double ratio = rt / c.rho0;
            const double pw = c.exponent_is_int ? powi(ratio, (long)c.gamma) : pow(ratio, c.gamma);
            pres = fmax(c.B * (pw - 1.0), 0.0);
        } else if (dp) {
            dp_adapt(c, stt);
        }
    }
    // advect_pos (eng/solver_sph_base.py:224-238; the XSPH sums are in aux3)
    if (ops & OP_POS) {
        for (int d = 0; d < 3; ++d) {
            x[d] = xsph ? x[d] + c.dt * (v[d] + 0.5 * xs[d]) : x[d] + c.dt * v[d];
            bad = bad || !isfinite(x[d]);
        }
    }
    // advect_something (the solvers' post-steps)
    int flag = 0;
    if (post) {
        rho = fmax(c.rho0, rho);
        mV = mass / rho;
        if (SOIL) {
            eq += c.dt * deq;
            if (dp) {
                flag = dp_flag(c, st);
                dp_adapt(c, st);
                eqp += c.dt * deqp;
            }
        }
    }

    if (bad) atomicOr(err, TSG_ERR_NONFINITE);
    if (upd_rho || post) p.density[i] = rho;
    if ((ops & (OP_HALF | OP_RK_STAGE)) || upd_rho || post) p.m_V[i] = mV;
    if (upd_rho) st3(p.v, v, n, i);
    if (ops & OP_POS) st3(p.x, x, n, i);
    if (ops & (OP_INIT | OP_HALF | OP_RK_STAGE)) { t.density_tmp[i] = rt; st3(t.v_tmp, vt, n, i); }
    if (ops & (OP_RK_INIT | OP_RK_UPDATE)) { t.d_density_RK[i] = ad; st3(t.d_vel_RK, av, n, i); }
    if (pre && !SOIL) {
        p.pressure[i] = pres;
        wc_record(c, pr.rec, i, vt, pres, rt, mV, ti == MAT_FLUID);
    }
    if (SOIL && soil) {
        if (pre && dp) soil_record(c, pr.rec, i, vt, stt, rt, mV);
        if ((ops & OP_INIT) || (dp && ((ops & (OP_HALF | OP_RK_STAGE)) || pre))) st9(t.stress_tmp, stt, n, i);
        if (dp && (ops & (OP_RK_INIT | OP_RK_UPDATE))) st9(t.d_stress_RK, as, n, i);
        if (dp && (upd_rho || post)) st9(p.stress, st, n, i);
        if (post) {
            p.strain_equ[i] = eq;
            if (dp) { p.strain_equ_p[i] = eqp; p.flag_retmap[i] = flag; }
        }
    }
}

// ---- enforce_boundary (eng/solver_sph_base.py:525-601) ----
__global__ void k_enforce(Consts c, Persist64 p) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    const int n = c.n;
    const int ti = p.mat_type[i];
    const bool rigid_dyn = ti == MAT_RIGID && p.is_dynamic[i];
    const bool on = c.boundary == 1 ? (is_flow(ti) || rigid_dyn) : rigid_dyn;
    if (!on) return;
    double pos[3], nrm[3] = {0, 0, 0};
    for (int d = 0; d < 3; ++d) pos[d] = p.x[(size_t)d * n + i];
    const double r = c.r_eps;
    if (pos[0] > c.de[0] - r) { nrm[0] += 1.0; p.x[i] = c.de[0] - r; }
    if (pos[0] <= c.ds[0] + r) { nrm[0] += -1.0; p.x[i] = c.ds[0] + r; }
    if (pos[1] <= c.ds[1] + r) { nrm[1] += -1.0; p.x[(size_t)n + i] = c.ds[1] + r; }
    if (c.dim == 3) {
        if (pos[2] > c.de[2] - r) { nrm[2] += 1.0; p.x[2 * (size_t)n + i] = c.de[2] - r; }
        if (pos[2] <= c.ds[2] + r) { nrm[2] += -1.0; p.x[2 * (size_t)n + i] = c.ds[2] + r; }
    }
    double ln = sqrt((nrm[0] * nrm[0] + nrm[1] * nrm[1]) + nrm[2] * nrm[2]);
    if (ln > EPS) {
        double u[3] = {nrm[0] / ln, nrm[1] / ln, nrm[2] / ln};
        double v[3];
        for (int d = 0; d < 3; ++d) v[d] = p.v[(size_t)d * n + i];
        double vd = (v[0] * u[0] + v[1] * u[1]) + v[2] * u[2];
        for (int d = 0; d < 3; ++d) p.v[(size_t)d * n + i] = v[d] - (1.0 + 0.3) * vd * u[d];
    }
}

// ---- inspection: neighbour lists in traversal order ----
template <int DIM>
__global__ void k_nbr_count(Consts c, Persist64 p, Trans64 t, const int* __restrict__ cs, int* counts) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    double xi[3];
    load_x<DIM>(p.x, i, c.n, xi);
    int m = 0;
    for_neighbors<DIM>(c, p.x, t.pos32, cs, i, xi, true, [&](int, const double*, double) { ++m; });
    counts[i] = m;
}

template <int DIM>
__global__ void k_nbr_fill(Consts c, Persist64 p, Trans64 t, const int* __restrict__ cs,
                           const int* __restrict__ offsets, int* list) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    double xi[3];
    load_x<DIM>(p.x, i, c.n, xi);
    int m = offsets[i];
    for_neighbors<DIM>(c, p.x, t.pos32, cs, i, xi, true, [&](int j, const double*, double) { list[m++] = j; });
}

// ---- FP64 diagnostics over flow particles ----
__device__ __forceinline__ void atomic_max_double(double* addr, double v) {
    unsigned long long* a = reinterpret_cast<unsigned long long*>(addr);
    unsigned long long old = *a;
    while (__longlong_as_double(old) < v) {
        unsigned long long prev = atomicCAS(a, old, __double_as_longlong(v));
        if (prev == old) break;
        old = prev;
    }
}

__global__ void k_diag(Consts c, Persist64 p, double* out) {
    __shared__ double sh[8][TPB / 32];
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = c.n;
    double v[8] = {0, 0, 0, 0, 0, 0, 0, -DBL_MAX};
    if (i < n && is_flow(p.mat_type[i])) {
        double m = p.mass[i];
        double vx = p.v[i], vy = p.v[(size_t)n + i], vz = p.v[2 * (size_t)n + i];
        double v2 = (vx * vx + vy * vy) + vz * vz;
        v[0] = m;
        v[1] = m * vx; v[2] = m * vy; v[3] = m * vz;
        v[4] = 0.5 * m * v2;
        v[5] = -m * ((c.g[0] * p.x[i] + c.g[1] * p.x[(size_t)n + i]) + c.g[2] * p.x[2 * (size_t)n + i]);
        v[6] = sqrt(v2);
        v[7] = p.x[i];
    }
    for (int o = 16; o > 0; o >>= 1) {
        for (int q = 0; q < 6; ++q) v[q] += __shfl_down_sync(0xffffffffu, v[q], o);
        v[6] = fmax(v[6], __shfl_down_sync(0xffffffffu, v[6], o));
        v[7] = fmax(v[7], __shfl_down_sync(0xffffffffu, v[7], o));
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) for (int q = 0; q < 8; ++q) sh[q][wid] = v[q];
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < TPB / 32; ++w) {
            for (int q = 0; q < 6; ++q) v[q] += sh[q][w];
            v[6] = fmax(v[6], sh[6][w]);
            v[7] = fmax(v[7], sh[7][w]);
        }
        for (int q = 0; q < 6; ++q) atomicAdd(&out[q], v[q]);
        atomic_max_double(&out[6], v[6]);
        atomic_max_double(&out[7], v[7]);
    }
}

__global__ void k_geostatic(Consts c, Persist64 p, const double* ymax_in, double K0) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    if (p.mat_type[i] != MAT_SOIL) return;
    const int n = c.n;
    double vs = c.rho0 * c.g[1] * (ymax_in[0] - p.x[(size_t)n + i]);
    p.stress[i] = K0 * vs;
    p.stress[4 * (size_t)n + i] = vs;
    p.stress[8 * (size_t)n + i] = K0 * vs;
}

__global__ void k_ymax_soil(Consts c, Persist64 p, double* out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    double y = -DBL_MAX;
    if (i < c.n && p.mat_type[i] == MAT_SOIL) y = p.x[(size_t)c.n + i];
    for (int o = 16; o > 0; o >>= 1) y = fmax(y, __shfl_down_sync(0xffffffffu, y, o));
    if ((threadIdx.x & 31) == 0) atomic_max_double(out, y);
}

}  // namespace

// ---------------------------------------------------------------- launchers
// ---- dynamic rigid bodies (eng/solver_sph_base.py:467-518) ----
// The reaction on dynamic rigid particles.  The reference subtracts every flow particle's
// pair term from its dynamic rigid neighbour inside the flow particle's loop
// (`pt[j].d_vel -= tmp`, eng/solver_sph_wc.py:70-71, eng/solver_sph_muI.py:45-46,
// eng/solver_sph_dp.py:164-165), an unsynchronised scatter.  Here every rigid particle
// gathers the terms of its flow neighbours in its own traversal order, which is ascending
// particle index (the serial order of the scatter), evaluating each term exactly as the flow
// particle's loop does (r = x_flow - x_rigid is the exact negation of the traversal's
// offset), starting from the gravity the boundary pass set.
template <int DIM>
__global__ void k_rigid_reaction(Consts c, Persist64 p, Trans64 t, const int* __restrict__ cs,
                                 const int* __restrict__ list, int count) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= count) return;
    const int j = list[k];
    if (!(p.mat_type[j] == MAT_RIGID && p.is_dynamic[j])) return;
    const int n = c.n;
    double xj[3];
    load_x<DIM>(p.x, j, n, xj);
    double dvj[3];
    for (int d = 0; d < 3; ++d) dvj[d] = t.d_vel[(size_t)d * n + j];
    const double mVj = p.m_V[j], rtj = t.density_tmp[j], ptj = p.pressure[j];
    double stj[9], vtj[3];
    if (c.solver != 1)
        for (int q = 0; q < 9; ++q) stj[q] = t.stress_tmp[(size_t)q * n + j];
    for (int d = 0; d < 3; ++d) vtj[d] = t.v_tmp[(size_t)d * n + j];
    for_neighbors<DIM>(c, p.x, t.pos32, cs, j, xj, true, [&](int i, const double* rji, double rn) {
        if (p.mat_type[i] != c.flow_type) return;
        double r[3] = {-rji[0], -rji[1], -rji[2]};
        if (DIM == 2) r[2] = 0.0;
        double kd[3], f[3] = {0.0, 0.0, 0.0};
        kernel_dW<DIM>(c, r, rn, kd);
        const double rti = t.density_tmp[i];
        if (c.solver == 1) {
            double dvv[3];
            for (int d = 0; d < DIM; ++d) dvv[d] = t.v_tmp[(size_t)d * n + i] - vtj[d];
            const double pri = p.pressure[i] / (rti * rti);
            wc_force_pair<DIM>(c, MAT_RIGID, mVj, dvv, rti, pri, ptj, rtj, r, rn, kd, f);
        } else {
            double kc[3], sti[9];
            if (c.corr == 1) {
                double L[9];
                for (int q = 0; q < 9; ++q) L[q] = t.CSPM_L[(size_t)q * n + i];
                matvec_corr<DIM>(L, kd, kc, PlainMul());
            } else {
                kc[0] = kd[0]; kc[1] = kd[1]; kc[2] = kd[2];
            }
            for (int q = 0; q < 9; ++q) sti[q] = t.stress_tmp[(size_t)q * n + i];
            stress_div_val<DIM>(sti, rti * rti, stj, rtj, mVj, kc, f);
        }
        for (int d = 0; d < DIM; ++d) dvj[d] = dvj[d] - f[d];
    });
    for (int d = 0; d < 3; ++d) t.d_vel[(size_t)d * n + j] = dvj[d];
}

// Object slot of a dynamic rigid particle (-1 for any other), for the list builder.
struct RigidSlot64 {
    const int* mt;
    const int* dyn;
    const int* oid;
    const int* ids;
    int nobj;
    __device__ int operator()(int i) const {
        if (mt[i] != MAT_RIGID || !dyn[i]) return -1;
        const int id = oid[i];
        for (int o = 0; o < nobj; ++o)
            if (ids[o] == id) return o;
        return -1;
    }
};

// The object sums of the shape matching are serial sums in ascending particle order (the
// oracle's order, so that the results are bit-identical).  The block stages each chunk of
// kSMChunk particles' terms (products rounded as in the serial expression: this unit is
// compiled without contracted multiply-adds) in shared memory with all its threads, and
// one thread adds them in order: the dependent additions run from shared memory instead of
// behind one gather per particle.
constexpr int kSMChunk = 512;

// init_rigid_body / calc_rigid_rest_m (eng/solver_sph_base.py:467-470, :517-518): the rest
// centre of mass of every dynamic rigid object from the uploaded positions, summed in upload
// order (the object's list, built before the first sort), one block per object.
__global__ void __launch_bounds__(kSMChunk) k_rest_cm(Consts c, Persist64 p, Rigid64 rb) {
    __shared__ double buf[4][kSMChunk];
    const int o = blockIdx.x;
    const int* list = rb.list + rb.off[o];
    const int m = rb.off[o + 1] - rb.off[o];
    const int n = c.n;
    double cm[3] = {0.0, 0.0, 0.0}, sum_m = 0.0;
    for (int k0 = 0; k0 < m; k0 += kSMChunk) {
        const int k = k0 + threadIdx.x;
        if (k < m) {
            const int i = list[k];
            const double mi = p.mass[i];
            for (int d = 0; d < 3; ++d) buf[d][threadIdx.x] = mi * p.x[(size_t)d * n + i];
            buf[3][threadIdx.x] = mi;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            const int cnt = min(kSMChunk, m - k0);
            for (int q = 0; q < cnt; ++q) {
                for (int d = 0; d < 3; ++d) cm[d] = cm[d] + buf[d][q];
                sum_m += buf[3][q];
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int d = 0; d < 3; ++d) rb.rest_cm[3 * o + d] = cm[d] / sum_m;
}

// solve_constraints (eng/solver_sph_base.py:478-500), one block per dynamic rigid object,
// over its list (ascending particle order, rebuilt after every sort): the centre of mass
// (calc_cm, :502-511) and A = sum (m_V rho p) q^T (p = x - cm, q = x0 - rest cm), both
// summed in list order, R = polar(A) (identity when every entry is below 1e-8), and finally
// every particle x += (cm + R q) - x.
__global__ void __launch_bounds__(kSMChunk) k_shape_match(Consts c, Persist64 p, Rigid64 rb) {
    __shared__ double buf[9][kSMChunk];
    __shared__ double cm_s[3], R_s[9];
    const int o = blockIdx.x;
    const int* list = rb.list + rb.off[o];
    const int m = rb.off[o + 1] - rb.off[o];
    const int n = c.n;
    double acc[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    double sum_m = 0.0;
    for (int k0 = 0; k0 < m; k0 += kSMChunk) {
        const int k = k0 + threadIdx.x;
        if (k < m) {
            const int i = list[k];
            const double mi = p.mass[i];
            for (int d = 0; d < 3; ++d) buf[d][threadIdx.x] = mi * p.x[(size_t)d * n + i];
            buf[3][threadIdx.x] = mi;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            const int cnt = min(kSMChunk, m - k0);
            for (int q = 0; q < cnt; ++q) {
                for (int d = 0; d < 3; ++d) acc[d] = acc[d] + buf[d][q];
                sum_m += buf[3][q];
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int d = 0; d < 3; ++d) cm_s[d] = acc[d] / sum_m;
    __syncthreads();
    for (int q = 0; q < 9; ++q) acc[q] = 0.0;
    for (int k0 = 0; k0 < m; k0 += kSMChunk) {
        const int k = k0 + threadIdx.x;
        if (k < m) {
            const int i = list[k];
            const double sc = p.m_V[i] * p.density[i];
            double sp[3], q[3];
            for (int d = 0; d < 3; ++d) {
                q[d] = p.x0[(size_t)d * n + i] - rb.rest_cm[3 * o + d];
                sp[d] = sc * (p.x[(size_t)d * n + i] - cm_s[d]);
            }
            for (int a = 0; a < 3; ++a)
                for (int b = 0; b < 3; ++b) buf[3 * a + b][threadIdx.x] = sp[a] * q[b];
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            const int cnt = min(kSMChunk, m - k0);
            for (int q = 0; q < cnt; ++q)
                for (int e = 0; e < 9; ++e) acc[e] = acc[e] + buf[e][q];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        double R[9];
        polar3(acc, R);
        bool small = true;
        for (int q = 0; q < 9; ++q) small = small && fabs(R[q]) < EPS;
        if (small)
            for (int q = 0; q < 9; ++q) R[q] = (q % 4 == 0) ? 1.0 : 0.0;
        for (int q = 0; q < 9; ++q) R_s[q] = R[q];
    }
    __syncthreads();
    for (int k = threadIdx.x; k < m; k += blockDim.x) {
        const int i = list[k];
        double q[3];
        for (int d = 0; d < 3; ++d) q[d] = p.x0[(size_t)d * n + i] - rb.rest_cm[3 * o + d];
        for (int a = 0; a < 3; ++a) {
            const double rq = (R_s[3 * a] * q[0] + R_s[3 * a + 1] * q[1]) + R_s[3 * a + 2] * q[2];
            const double goal = cm_s[a] + rq;
            const double xa = p.x[(size_t)a * n + i];
            const double corr = (goal - xa) * 1.0;
            p.x[(size_t)a * n + i] = xa + corr;
        }
    }
}

static void rigid_lists64(const Consts& c, const Persist64& p, const Rigid64& r, cudaStream_t s) {
    build_rigid_lists(c.n, r.nobj, RigidSlot64{p.mat_type, p.is_dynamic, p.obj_id, r.obj_id, r.nobj}, r.scratch,
                      r.off, r.list, s);
}

#define DISPATCH_DIM(c, KERNEL, GRID, ...)                                   \
    do {                                                                     \
        if ((c).dim == 2) TSG_LAUNCH(KERNEL<2>, GRID, TPB, s, __VA_ARGS__);       \
        else TSG_LAUNCH(KERNEL<3>, GRID, TPB, s, __VA_ARGS__);                    \
    } while (0)

// Lanes per row: four, about as many as a loop has sums (2 to 5 in most), so that the additions
// in slot order cost what one thread's would (8 lanes: 3D, 118 k rows, 4,203 us a step against
// 2,819; 2D mu(I), 20 k rows, 216 against 187); eight in 2D scenes whose rows leave the SMs
// short of warps, where the loop is a chain of latencies (7.2 k rows: 905 us per ten steps
// against 1,091; 600 rows: 75 us a step against 86; 16 lanes lose at both).
// The line: 8 x 8,192 threads are a quarter of what the GPU holds.  3D rows have four times the
// entries to share out and keep four.
constexpr int LANES = 4, LANES_SMALL = 8, SMALL_ROWS = 8192;
inline bool small_rows(const Consts& c) { return c.dim == 2 && c.n_flow <= SMALL_ROWS; }
inline int nrows(int count) { return (count + ROWS - 1) / ROWS; }
// Threads of a row kernel: without rows only the epilogue's threads have work.
inline int row_threads(const Grid& g, int lanes) { return g.pr.cap_f ? ROWS * lanes : ROWS; }

#define ROWS_LAUNCH(g, LN, COUNT, KERNEL, ...) TSG_LAUNCH(KERNEL, nrows(COUNT), row_threads(g, LN), s, __VA_ARGS__)
#define DISPATCH_ROWS(c, g, KERNEL, COUNT, ...)                                                            \
    do {                                                                                                   \
        if (small_rows(c)) ROWS_LAUNCH(g, LANES_SMALL, COUNT, (KERNEL<2, LANES_SMALL>), __VA_ARGS__);      \
        else if ((c).dim == 2) ROWS_LAUNCH(g, LANES, COUNT, (KERNEL<2, LANES>), __VA_ARGS__);              \
        else ROWS_LAUNCH(g, LANES, COUNT, (KERNEL<3, LANES>), __VA_ARGS__);                                \
    } while (0)
#define DISPATCH_ROWS_B(c, g, KERNEL, FLAG, COUNT, ...)                                                        \
    do {                                                                                                       \
        if (small_rows(c)) ROWS_LAUNCH(g, LANES_SMALL, COUNT, (KERNEL<2, LANES_SMALL, FLAG>), __VA_ARGS__);    \
        else if ((c).dim == 2) ROWS_LAUNCH(g, LANES, COUNT, (KERNEL<2, LANES, FLAG>), __VA_ARGS__);            \
        else ROWS_LAUNCH(g, LANES, COUNT, (KERNEL<3, LANES, FLAG>), __VA_ARGS__);                              \
    } while (0)
#define DISPATCH_KC(c, g, KERNEL, MODE, COUNT, ...)                                                 \
    do {                                                                                            \
        if ((MODE) == KC_READ) DISPATCH_ROWS_B(c, g, KERNEL, KC_READ, COUNT, __VA_ARGS__);          \
        else if ((MODE) == KC_KEEP) DISPATCH_ROWS_B(c, g, KERNEL, KC_KEEP, COUNT, __VA_ARGS__);     \
        else DISPATCH_ROWS_B(c, g, KERNEL, KC_MAKE, COUNT, __VA_ARGS__);                            \
    } while (0)

static void build_rows(const Consts& c, const Persist64& p, const Trans64& t, const Grid& g, bool flow_only,
                       bool sorted, cudaStream_t s) {
    if (!g.pr.cap_f) return;
    const int nb = flow_only ? 0 : c.n_bdy;
    const int rows = c.n_flow + nb;
    if (rows <= 0) return;
    const unsigned char* cf = sorted ? g.cell_flow : nullptr;
    const auto launch = [&](auto* k, int rpw) {
        TSG_LAUNCH(k, (rows + 8 * rpw - 1) / (8 * rpw), 256, s, c, p.x, t.pos32, t.pos32l, t.cell0, g.cell_start, cf,
                   g.list_flow, c.n_flow, g.list_bdy, nb, flow_only, g.pr);
    };
    // Three rows a warp share one look-up of their 27 ranges (most boundary rows are empty), but
    // leave a third of the warps.  3D, us per step with one and three: 28 k rows 276 / 280, 76 k
    // 398 / 398, 141 k 696 / 691, 476 k 2,770 / 2,738.
    if (c.dim == 2) launch(k_list64<2, 1>, 1);
    else if (rows < 98304) launch(k_list64<3, 1>, 1);
    else launch(k_list64<3, 3>, 3);
}

void fp64_build_rows(const Consts& c, const Persist64& p, const Trans64& t, const Grid& g, bool sorted,
                     cudaStream_t s) {
    PhaseScope ph(s, PH_LISTS);
    build_rows(c, p, t, g, false, sorted, s);
}

void fp64_geometry(const Consts& c, const Persist64& p, Trans64& t, const Grid& g, cudaStream_t s) {
    if (!g.pr.cap_f) return;
    PhaseScope ph(s, PH_LISTS);
    if (c.n_flow > 0) DISPATCH_ROWS(c, g, k_geom_flow, c.n_flow, c, p, g.list_flow, c.n_flow, g.pr);
    if (c.n_bdy > 0) DISPATCH_ROWS(c, g, k_geom_bdy, c.n_bdy, c, p, g.list_bdy, c.n_bdy, g.pr);
}

// Block size of the per-particle passes: small scenes in blocks of one warp, to reach every SM.
static int tpb(int n) { return n < 152 * 4 * TPB ? 32 : TPB; }

static void particle_pass(const Consts& c, const Persist64& p, const Trans64& t, const Grid& g, unsigned ops, int m,
                          cudaStream_t s) {
    if (c.solver == 2) ops &= ~(unsigned)OP_PRE;
    if (!ops) return;
    PhaseScope ph(s, ops & (OP_HALF | OP_RK_STAGE | OP_RK_UPDATE | OP_FULL | OP_RK_FINAL | OP_RK_INIT) ? PH_INTEGRATE
                     : ops & OP_INIT ? PH_INIT : ops & OP_PRE ? PH_PRE : ops & OP_POS ? PH_POS : PH_POST);
    if (c.solver == 1) TSG_LAUNCH(k_particle<false>, nblk(c.n, tpb(c.n)), tpb(c.n), s, c, p, t, g.pr, ops, m, g.err);
    else TSG_LAUNCH(k_particle<true>, nblk(c.n, tpb(c.n)), tpb(c.n), s, c, p, t, g.pr, ops, m, g.err);
}

static void corr_flow(const Consts& c, const Persist64& p, Trans64& t, const Grid& g, cudaStream_t s) {
    if (c.n_flow <= 0) return;
    PhaseScope ph(s, PH_CORR);
    if (c.corr == 1)
        DISPATCH_ROWS_B(c, g, k_corr_flow, true, c.n_flow, c, p, t, g.cell_start, g.list_flow, c.n_flow, g.pr);
    else
        DISPATCH_ROWS_B(c, g, k_corr_flow, false, c.n_flow, c, p, t, g.cell_start, g.list_flow, c.n_flow, g.pr);
}

static void corr_bdy(const Consts& c, const Persist64& p, Trans64& t, const Grid& g, cudaStream_t s) {
    if (c.n_bdy <= 0) return;
    PhaseScope ph(s, PH_CORR);
    DISPATCH_ROWS(c, g, k_corr_bdy, c.n_bdy, c, p, t, g.cell_start, g.list_bdy, c.n_bdy, g.pr);
}

void fp64_kernel_corr(const Consts& c, const Persist64& p, Trans64& t, const Grid& g, cudaStream_t s) {
    corr_flow(c, p, t, g, s);
    corr_bdy(c, p, t, g, s);
}

void fp64_rest_cm(const Consts& c, const Persist64& p, const Rigid64& r, cudaStream_t s) {
    if (r.nobj <= 0) return;
    rigid_lists64(c, p, r, s);
    TSG_LAUNCH(k_rest_cm, r.nobj, kSMChunk, s, c, p, r);
}

void fp64_solve_rigid(const Consts& c, Persist64& p, const Rigid64& r, cudaStream_t s) {
    if (r.nobj <= 0) return;
    PhaseScope ph(s, PH_POS);
    rigid_lists64(c, p, r, s);
    TSG_LAUNCH(k_shape_match, r.nobj, kSMChunk, s, c, p, r);
}

void fp64_density_sum(const Consts& c, const Persist64& p, const Trans64& t, const Grid& g, double* out,
                      cudaStream_t s) {
    PhaseScope ph(s, PH_OTHER);
    DISPATCH_DIM(c, k_density_sum, nblk(c.n), c, p, t, g.cell_start, out);
}

void fp64_init_tmp(const Consts& c, const Persist64& p, Trans64& t, const Grid& g, cudaStream_t s) {
    particle_pass(c, p, t, g, OP_INIT, 0, s);
}

// The loops of one_step after its per-particle first phase.  stage: how often this step's loops
// have run before (the first stores the corrected gradients for the others); -1: the only time.
// Without the correction the gradient is grad W itself: nothing to keep.
static int gradient_mode(const Consts& c, int stage) {
    return c.corr != 1 || stage < 0 ? KC_MAKE : stage == 0 ? KC_KEEP : KC_READ;
}

static void mui_stress(const Consts& c, Persist64& p, Trans64& t, const Grid& g, int stage, cudaStream_t s) {
    if (c.solver != 2 || c.n_flow <= 0) return;
    PhaseScope ph(s, PH_PRE);
    int kc = gradient_mode(c, stage);
    if (c.corr == 1 && kc == KC_MAKE) kc = KC_KEEP;  // the momentum loop reads it
    DISPATCH_KC(c, g, k_mui_stress, kc, c.n_flow, c, p, t, g.cell_start, g.list_flow, c.n_flow, g.pr);
}

static void bdy(const Consts& c, Persist64& p, Trans64& t, const Grid& g, cudaStream_t s) {
    if (c.n_bdy <= 0) return;
    PhaseScope ph(s, PH_BDY);
    if (c.solver == 1) DISPATCH_ROWS_B(c, g, k_bdy, false, c.n_bdy, c, p, t, g.cell_start, g.list_bdy, c.n_bdy, g.pr);
    else DISPATCH_ROWS_B(c, g, k_bdy, true, c.n_bdy, c, p, t, g.cell_start, g.list_bdy, c.n_bdy, g.pr);
}

static void rates(const Consts& c, Persist64& p, Trans64& t, const Grid& g, int stage, cudaStream_t s) {
    if (c.n_flow > 0) {
        PhaseScope ph(s, PH_RATES);
        const int kc = gradient_mode(c, stage);
        if (c.solver == 1)
            DISPATCH_KC(c, g, k_wc_rates, kc, c.n_flow, c, p, t, g.cell_start, g.list_flow, c.n_flow, g.pr);
        else if (c.solver == 2 && c.corr == 1)
            DISPATCH_ROWS_B(c, g, k_mui_mom, KC_READ, c.n_flow, c, p, t, g.cell_start, g.list_flow, c.n_flow, g.pr);
        else if (c.solver == 2)
            DISPATCH_ROWS_B(c, g, k_mui_mom, KC_MAKE, c.n_flow, c, p, t, g.cell_start, g.list_flow, c.n_flow, g.pr);
        else
            DISPATCH_KC(c, g, k_dp_rates, kc, c.n_flow, c, p, t, g.cell_start, g.list_flow, c.n_flow, g.pr);
    }
    if (c.n_rigid_dyn > 0 && c.n_bdy > 0) {  // the flow's reaction on dynamic rigid particles
        PhaseScope ph(s, PH_RATES);
        DISPATCH_DIM(c, k_rigid_reaction, nblk(c.n_bdy), c, p, t, g.cell_start, g.list_bdy, c.n_bdy);
    }
}

void fp64_one_step(const Consts& c, Persist64& p, Trans64& t, const Grid& g, cudaStream_t s) {
    particle_pass(c, p, t, g, OP_PRE, 0, s);
    mui_stress(c, p, t, g, -1, s);
    bdy(c, p, t, g, s);
    rates(c, p, t, g, -1, s);
}

static void xsph(const Consts& c, const Persist64& p, Trans64& t, const Grid& g, cudaStream_t s) {
    if (!c.xsph) return;
    PhaseScope ph(s, PH_POS);
    if (c.n_flow > 0) DISPATCH_ROWS(c, g, k_xsph, c.n_flow, c, p, t, g.cell_start, g.list_flow, c.n_flow, g.pr);
    if (c.n_rigid_dyn > 0) DISPATCH_DIM(c, k_xsph_rigid, nblk(c.n_bdy), c, p, t, g.cell_start, g.list_bdy, c.n_bdy);
}

// mu(I): what follows the per-particle part of advect_something.
static void mui_regularise(const Consts& c, Persist64& p, Trans64& t, const Grid& g, cudaStream_t s) {
    if (c.solver != 2 || c.n_flow <= 0) return;
    PhaseScope ph(s, PH_POST);
    if (g.pr.cap_f) fp64_refresh_pos32(c, p, t, s);
    build_rows(c, p, t, g, true, false, s);
    DISPATCH_ROWS(c, g, k_post_mui, c.n_flow, c, p, t, g.cell_start, g.list_flow, c.n_flow, g.pr);
}

// substep by the integrator, from the per-particle first phase of its first loops (run by the
// caller) to its last update, which `tail` follows in the same launch.  first_bdy: the first
// boundary loop is still to run.
static void substep_loops(const Consts& c, Persist64& p, Trans64& t, const Grid& g, unsigned tail, bool first_bdy,
                          cudaStream_t s) {
    auto loops = [&](int stage, bool with_bdy) {
        mui_stress(c, p, t, g, stage, s);
        if (with_bdy) bdy(c, p, t, g, s);
        rates(c, p, t, g, stage, s);
    };
    if (c.ti == 1) {
        loops(-1, first_bdy);
        particle_pass(c, p, t, g, OP_FULL | tail, 0, s);
    } else if (c.ti == 2) {
        loops(0, first_bdy);
        particle_pass(c, p, t, g, OP_HALF | OP_PRE, 0, s);
        loops(1, true);
        particle_pass(c, p, t, g, OP_FULL | tail, 0, s);
    } else {
        const int m[4] = {1, 2, 2, 1};
        for (int k = 0; k < 4; ++k) {
            loops(k, k > 0 || first_bdy);
            particle_pass(c, p, t, g, OP_RK_UPDATE | (k < 3 ? OP_RK_STAGE | OP_PRE : OP_RK_FINAL | tail), m[k], s);
        }
    }
}
static unsigned substep_head(const Consts& c) { return (c.ti == 4 ? OP_RK_INIT : 0u) | OP_PRE; }

void fp64_substep(const Consts& c, Persist64& p, Trans64& t, const Grid& g, cudaStream_t s) {
    particle_pass(c, p, t, g, substep_head(c), 0, s);
    substep_loops(c, p, t, g, 0, true, s);
}

void fp64_step(const Consts& c, Persist64& p, Trans64& t, const Grid& g, const Rigid64& r, bool collide,
               cudaStream_t s) {
    fp64_build_rows(c, p, t, g, true, s);
    // The correction pass over the flow rows and what the first rates loop needs besides (the
    // per-particle start, the boundary rows' Shepard factors and extrapolation) touch different
    // arrays: two branches of the graph (a small scene fills neither the GPU nor a launch's
    // latency with one of them).  mu(I) extrapolates after its stress loop.
    const bool early_bdy = c.solver != 2;
    Fork branches;
    corr_flow(c, p, t, g, s);
    branches.second();
    particle_pass(c, p, t, g, OP_INIT | substep_head(c), 0, s);
    corr_bdy(c, p, t, g, s);
    if (early_bdy) bdy(c, p, t, g, s);
    branches.join();
    substep_loops(c, p, t, g, c.xsph ? 0u : OP_POS | OP_POST, !early_bdy, s);
    if (c.xsph) {
        xsph(c, p, t, g, s);
        particle_pass(c, p, t, g, OP_POS | OP_POST, 0, s);
    }
    mui_regularise(c, p, t, g, s);
    if (c.n_rigid_dyn) fp64_solve_rigid(c, p, r, s);
    // enforce_boundary also clamps dynamic rigid particles in every boundary mode
    if (collide || c.n_rigid_dyn) fp64_advect(c, p, t, g, TSG_ENFORCE_BOUNDARY, s);
}

void fp64_advect(const Consts& c, Persist64& p, Trans64& t, const Grid& g, int which, cudaStream_t s) {
    switch (which) {
    case TSG_ADVECT_FULL: particle_pass(c, p, t, g, OP_FULL, 0, s); break;
    case TSG_ADVECT_LF_HALF: particle_pass(c, p, t, g, OP_HALF, 0, s); break;
    case TSG_ADVECT_POS:
        xsph(c, p, t, g, s);
        particle_pass(c, p, t, g, OP_POS, 0, s);
        break;
    case TSG_ADVECT_SOMETHING:
        particle_pass(c, p, t, g, OP_POST, 0, s);
        mui_regularise(c, p, t, g, s);
        break;
    case TSG_ENFORCE_BOUNDARY: {
        PhaseScope ph(s, PH_OTHER);
        TSG_LAUNCH(k_enforce, nblk(c.n), TPB, s, c, p);
        break;
    }
    case TSG_RK_INIT: particle_pass(c, p, t, g, OP_RK_INIT, 0, s); break;
    case TSG_RK_STAGE: particle_pass(c, p, t, g, OP_RK_STAGE, 0, s); break;
    case TSG_RK_FINAL: particle_pass(c, p, t, g, OP_RK_FINAL, 0, s); break;
    default: break;
    }
}

void fp64_rk_update(const Consts& c, Persist64& p, Trans64& t, const Grid& g, int m, cudaStream_t s) {
    particle_pass(c, p, t, g, OP_RK_UPDATE, m, s);
}

void fp64_neighbors(const Consts& c, const Persist64& p, const Trans64& t, const Grid& g,
                    int* counts, int* offsets, int* list, cudaStream_t s) {
    if (!list) {
        DISPATCH_DIM(c, k_nbr_count, nblk(c.n), c, p, t, g.cell_start, counts);
    } else {
        DISPATCH_DIM(c, k_nbr_fill, nblk(c.n), c, p, t, g.cell_start, offsets, list);
    }
}

void fp64_diag(const Consts& c, const Persist64& p, double* out8, cudaStream_t s) {
    double init[8] = {0, 0, 0, 0, 0, 0, 0, -DBL_MAX};
    cudaMemcpyAsync(out8, init, sizeof init, cudaMemcpyHostToDevice, s);
    cudaStreamSynchronize(s);
    TSG_LAUNCH(k_diag, nblk(c.n), TPB, s, c, p, out8);
}

void fp64_init_geostatic(const Consts& c, Persist64& p, double* scratch, cudaStream_t s) {
    double init = -DBL_MAX;
    cudaMemcpyAsync(scratch, &init, sizeof init, cudaMemcpyHostToDevice, s);
    cudaStreamSynchronize(s);
    TSG_LAUNCH(k_ymax_soil, nblk(c.n), TPB, s, c, p, scratch);
    TSG_LAUNCH(k_geostatic, nblk(c.n), TPB, s, c, p, scratch, c.K0);
}

__global__ void k_refresh_pos32_impl(Consts c, const double* __restrict__ x, const int* __restrict__ mt,
                                     float4* __restrict__ pos32, float4* __restrict__ pos32l,
                                     long long* __restrict__ cell0) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    const size_t n = c.n;
    const double xi[3] = {x[i], x[n + i], x[2 * n + i]};
    write_pos32(c, xi, is_flow(mt[i]), pos32 + i, pos32l + i);
    cell0[i] = flat_cell(c, xi);
}

void fp64_refresh_pos32(const Consts& c, const Persist64& p, Trans64& t, cudaStream_t s) {
    TSG_LAUNCH(k_refresh_pos32_impl, nblk(c.n), TPB, s, c, p.x, p.mat_type, t.pos32, t.pos32l, t.cell0);
}

}  // namespace tsg
