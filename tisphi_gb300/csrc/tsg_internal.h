// Internal declarations shared by the CUDA translation units of libtisphi_gb300.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <tuple>
#include <utility>
#include <vector>

#include "../../include/tisphi_gb300.h"

namespace tsg {

// Host-side count of kernel launches issued by this library (all handles).  Graph replays
// add their kernel-node counts through add_launches.
void note_launch();
void add_launches(long long delta);
long long launch_total();
// True while tsg_profile is on (steps then run eagerly, with per-phase events).
bool profiling_on();

// A graph under construction on the calling thread: while one is set (Recording), launches and
// copies are added to it as nodes, each after the one before, instead of going to their stream.
// Not a stream capture: while one is open anywhere in the process, a device-wide
// synchronisation on any other thread fails and breaks the capture, and what the capturing
// thread launches after that runs at once.
struct Tape {
    cudaGraph_t graph;
    std::vector<cudaGraphNode_t> deps;  // what the next node waits for
    long long kernels = 0;
    bool ok = true;
    explicit Tape(cudaGraph_t g) : graph(g) {}
    template <class... P, class... A>
    void launch(void (*f)(P...), dim3 grid, dim3 block, A&&... a) {
        std::tuple<P...> v(std::forward<A>(a)...);
        std::apply([&](auto&... x) {
            void* args[] = {&x...};
            node(reinterpret_cast<void*>(f), grid, block, args);
        }, v);
    }
    void node(void* f, dim3 grid, dim3 block, void** args);
    void zero(void* p, size_t bytes);
    void copy(void* dst, const void* src, size_t bytes);
    void added(cudaError_t e, cudaGraphNode_t n);
};
Tape*& tape();
struct Recording {
    Tape* outer;
    explicit Recording(Tape& t) : outer(tape()) { tape() = &t; }
    ~Recording() { tape() = outer; }
};
// Two branches of a graph from here on; launched eagerly, one after the other.
struct Fork {
    std::vector<cudaGraphNode_t> from, first;
    Fork() { if (tape()) from = tape()->deps; }
    void second() { if (tape()) { first = tape()->deps; tape()->deps = from; } }
    void join();
};
// While it lives, this thread may make and destroy graphs although another thread
// captures a stream in the default (global) mode; without it the first such call fails and breaks
// that capture.
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    RelaxedCapture(const RelaxedCapture&) = delete;
};
// Device memory set to zero, or copied on the device, in stream order.
void zero_async(void* p, size_t bytes, cudaStream_t s);
void copy_async(void* dst, const void* src, size_t bytes, cudaStream_t s);

#define TSG_LAUNCH(kernel, grid, block, stream, ...)                       \
    do {                                                                    \
        if (::tsg::Tape* tape_ = ::tsg::tape()) {                           \
            tape_->launch(kernel, dim3(grid), dim3(block), __VA_ARGS__);    \
        } else {                                                            \
            ::tsg::note_launch();                                           \
            kernel<<<(grid), (block), 0, (stream)>>>(__VA_ARGS__);          \
        }                                                                   \
    } while (0)

// Phase profiling: when enabled, every launcher brackets its kernels with CUDA events
// recorded on the launching stream, and elapsed times are summed per phase.
enum Phase { PH_SORT = 0, PH_CORR, PH_INIT, PH_PRE, PH_BDY, PH_RATES, PH_INTEGRATE, PH_POS, PH_POST, PH_OTHER, PH_LISTS, PH_COUNT };
struct PhaseScope {
    PhaseScope(cudaStream_t s, int phase);
    ~PhaseScope();
    cudaStream_t s_;
    int phase_;
    void* stop_;
};

constexpr int MAT_REP = -2, MAT_DUMMY = -1, MAT_FLUID = 1, MAT_SOIL = 2, MAT_RIGID = 11;
constexpr double EPS = 1e-8;      // SPHBase.epsilon (eng/solver_sph_base.py:25)
constexpr double EPS_F = 1e-4;    // DPSPHSolver.eps_f (eng/solver_sph_dp.py:23)

// Scene constants derived on the host once, passed to every kernel by value.
struct Consts {
    int dim, solver, kernel, corr, xsph, boundary, exponent_is_int, ti;
    int n, n_flow, n_bdy, flow_type;
    int gnum[3];
    long long G;
    double vs[3], grid, R, h, h1, kk, visc_fac, eps_h2, h2;
    double rho0, B, gamma, dt, hdt, dt6, g[3];
    double mu, vsound2, coh;
    double alpha, k_c, kc_over_alpha, Gm, Km, sin_dila, lam_den, three_aK, nine_K_sin, twoG;
    double damp_E, damp_eps, K0;
    double rep_fac, diam, h075;
    double ds[3], de[3], r_eps;
    // f32 candidate prefilter: reject when |dx_f32|^2 > pf_r2; valid for centres with
    // every |x - vdomain_start| below pf_lim
    int pf_on;
    float pf_r2, pf_lim;
    float pf_in2;       // below this f32 distance^2 a pair is certainly a neighbour
    float pf_lo2, pf_hi2;  // the same two bounds for the distance^2 with the low parts added
    float cell_inv, cell_lim;  // 1 / cell size; support radius^2 in cells, widened (inf: cells are not tested)
    int kern_int;       // kernel constants inside 2^+-100 (int_mul chains stay normal)
    double kk6;         // kk / 6
    double rgrid;       // 1 / grid, and div_by's window for it
    unsigned grid_span;
    unsigned div_span;  // exponent window of div_by (0 closes it)
    double R2T;         // r2 < R2T exactly when sqrt(r2) < R
    int n_rigid_dyn;    // dynamic rigid particles (shape-matched bodies)
};

// Largest cell segment whose particles the reorder passes rank among themselves in scenes above
// kSortAll particles (larger ones: tsg_cellsort.cuh), and the size of the list of larger cells (at most n / (kSortSmall + 1) of them).
constexpr int kSortSmall = 256;
// Up to this many particles the reorder pass ranks every cell itself, however large
// (rank_in_cell), and the launch that orders the larger cells is left out.
constexpr int kSortAll = 16384;
inline int sort_small(int n) { return n <= kSortAll ? 0x7fffffff : kSortSmall; }
inline size_t cellsort_big_ints(long long n) { return (size_t)(n / kSortSmall + 2); }

// Block size of the rigid-object list builder (tsg_rigid_list.cuh) and its scratch size.
constexpr int kRListBlock = 256;
inline int rlist_blocks(int n) { return (n + kRListBlock - 1) / kRListBlock; }
inline size_t rlist_scratch_ints(int n, int nobj) { return (size_t)nobj * (size_t)rlist_blocks(n); }

// Dynamic rigid bodies (eng/solver_sph_base.py:467-518): object ids, rest centres of mass
// (from the uploaded positions, in upload order) and, per object, the slice of `list`
// that the list builder (tsg_rigid_list.cuh) fills with the object's particles in
// ascending order before every shape matching.
struct Rigid64 {
    int nobj = 0;
    int* obj_id = nullptr;      // nobj (device)
    double* rest_cm = nullptr;  // 3 nobj (device)
    int* off = nullptr;         // nobj + 1 (device): slice starts in list
    int* list = nullptr;        // n_rigid_dyn (device)
    int* scratch = nullptr;     // nobj * ceil(n / 256) (device): the list builder's block offsets
};

// Persistent per-particle fields (permuted by the sort; double-buffered).
struct Persist64 {
    double* x;          // 3 planes of n
    double* v;          // 3 planes
    double* x0;         // 3 planes
    double* density;
    double* mass;
    double* m_V;
    double* pressure;
    double* stress;     // 9 planes (soil solvers) or nullptr
    double* strain_equ;
    double* strain_equ_p;
    int* flag_retmap;
    int* mat_type;
    int* mat_id;
    int* obj_id;
    int* is_dynamic;
    int* id0;
};

// Transient per-particle fields (recomputed every step, in sorted order).
struct Trans64 {
    double* v_tmp;      // 3 planes
    double* density_tmp;
    double* stress_tmp; // 9 planes or nullptr
    double* d_density;
    double* d_vel;      // 3 planes
    double* d_stress;   // 9 planes or nullptr (DP)
    double* v_grad;     // 9 planes or nullptr (soil)
    double* CSPM_f;
    double* CSPM_L;     // 9 planes or nullptr (kernel_corr)
    double* d_strain_equ;
    double* d_strain_equ_p;
    double* d_density_RK;
    double* d_vel_RK;   // 3 planes
    double* d_stress_RK;// 9 planes or nullptr
    double* aux3;       // 3 planes: XSPH sums
    float4* pos32;      // (x - vdomain_start) as f32, candidate prefilter; w = 1 for flow particles
    float4* pos32l;     // what pos32 rounds off, as f32
    long long* cell0;   // flattened cell index of the position, kNoCell if it has none
};
constexpr long long kNoCell = (long long)1 << 62;

// Neighbour rows of the current positions (tsg_pairs64.cuh): row k of the flow block belongs to
// particle list_flow[k], row k of the boundary block to list_bdy[k].  Row-major with a fixed
// pitch (a multiple of 8 slots); a row whose count exceeds it is walked through the cells.
// cap_f == 0: no rows (not enough device memory), every particle walks the cells.
struct Pairs64 {
    int cap_f, cap_b;
    size_t slots_f;     // n_flow * cap_f: plane stride of gk
    int* cnt;           // n_flow + n_bdy
    int* nb_f;          // entries: particle index, sign bit set for a non-flow neighbour
    int* nb_b;
    double* gk;         // dim planes: kernel gradient of each flow entry
    double2* gden;      // |r|^2 + 0.01 h^2 of each flow entry and its divisor() bits (WCSPH)
    double* gc;         // dim planes: corrected gradient L_i grad W of each flow entry (CSPM);
                        // the soil solvers, which use no other gradient, keep it in gk
    double* gw;         // kernel value of each boundary entry
    double* rec;        // 8 doubles per particle (16 for 3D soil): what a rates loop reads of a neighbour
};

// Sort scratch and cell table.
struct Grid {
    int* cell_of;       // per particle (old order)
    int* rank;          // per particle within-cell arrival rank
    long long* cell0_old;  // per particle (old order): unclipped flattened cell index
    int* count;         // G + 1; zeroed with what follows it in one memory set per sort:
                        // list_count, nbig, cell_flow
    size_t zero_bytes;
    int* cell_start;    // G + 2 exclusive starts; [G] = out-of-grid bin, [G+1] = n
    int* perm;          // new -> old
    int* tile_sum;      // scan partials
    int* list_flow;     // flow particles (sorted indices)
    int* list_bdy;      // boundary + rigid particles
    int* list_count;    // [0] flow, [1] bdy
    int* err;           // device error word
    int* big;           // cells above kSortSmall particles (cellsort_big_ints)
    int* nbig;          // their count
    unsigned char* cell_flow;  // per cell: 1 if it holds flow particles (as of the last sort)
    Pairs64 pr;         // neighbour rows
};

// ---- headless visual buffer (tsg_visual.cu) ----
// Planar f64 / int views of the fields a colour title may read (null when absent).
struct VisFields {
    const double *x, *x0, *v, *d_vel, *v_tmp, *density, *d_density, *pressure, *stress, *strain_equ,
        *strain_equ_p, *CSPM_L;
    const int *id0, *mat_type, *flag;
    int n;
};
int visual_launch(const VisFields& f, const tsg_visual_cfg& vc, double* scratch, float* pos, float* col,
                  double* range_out, cudaStream_t s);

// ---- launchers (tsg_sort.cu) ----
void sort_fp64(const Consts& c, Persist64& cur, Persist64& nxt, Trans64& t, Grid& g, cudaStream_t s);
void scan_exclusive(const int* in, int* out, int n, int* tile_sum, cudaStream_t s);
// Counting sort between the hash and the reorder: cell_start from the counts, perm in arrival
// order inside the cells, the cells that the reorder pass does not rank ordered.
void sort_cells(int n, int nbins, const int* count, int* cell_start, int* tile_sum, const int* cell_of, const int* rank,
                int* perm, int* big, int* nbig, cudaStream_t s);

// ---- launchers (tsg_fp64.cu) ----
void fp64_kernel_corr(const Consts& c, const Persist64& p, Trans64& t, const Grid& g, cudaStream_t s);
// Neighbour rows of the current positions, and the pair geometry without the correction
// factors (for a loop called on its own; fp64_kernel_corr writes the geometry too).
// sorted: positions and types are those of the last sort (cell_flow holds).
void fp64_build_rows(const Consts& c, const Persist64& p, const Trans64& t, const Grid& g, bool sorted,
                     cudaStream_t s);
void fp64_geometry(const Consts& c, const Persist64& p, Trans64& t, const Grid& g, cudaStream_t s);
void fp64_init_tmp(const Consts& c, const Persist64& p, Trans64& t, const Grid& g, cudaStream_t s);
void fp64_one_step(const Consts& c, Persist64& p, Trans64& t, const Grid& g, cudaStream_t s);
// substep (its integrator's loops and updates) on current rows and geometry.
void fp64_substep(const Consts& c, Persist64& p, Trans64& t, const Grid& g, cudaStream_t s);
// A step after its sort.
void fp64_step(const Consts& c, Persist64& p, Trans64& t, const Grid& g, const Rigid64& r, bool collide,
               cudaStream_t s);
void fp64_advect(const Consts& c, Persist64& p, Trans64& t, const Grid& g, int which, cudaStream_t s);
void fp64_rk_update(const Consts& c, Persist64& p, Trans64& t, const Grid& g, int m, cudaStream_t s);
void fp64_neighbors(const Consts& c, const Persist64& p, const Trans64& t, const Grid& g,
                    int* counts, int* offsets, int* list, cudaStream_t s);
void fp64_diag(const Consts& c, const Persist64& p, double* out8, cudaStream_t s);
void fp64_solve_rigid(const Consts& c, Persist64& p, const Rigid64& r, cudaStream_t s);
void fp64_rest_cm(const Consts& c, const Persist64& p, const Rigid64& r, cudaStream_t s);
void fp64_density_sum(const Consts& c, const Persist64& p, const Trans64& t, const Grid& g, double* out,
                      cudaStream_t s);
void fp64_init_geostatic(const Consts& c, Persist64& p, double* scratch, cudaStream_t s);
void fp64_refresh_pos32(const Consts& c, const Persist64& p, Trans64& t, cudaStream_t s);

}  // namespace tsg
