// solver.cu -- the fea_solver handle and the C ABI of include/fea_gpu.h.
//
// A handle holds one mesh and plays the roles of the reference's FEMContext
// (mesh, idx_map, assembled matrices; src/FEM/FEMContext.cpp) and of a Solver
// implementation (state fields u, v and advance_time; include/FEM/Solver.hpp).
#include <algorithm>
#include <charconv>
#include <cstdio>
#include <unordered_map>
#include <cstdarg>
#include <cstring>
#include <new>
#include <utility>

#include "fea_internal.cuh"

namespace fea {

namespace {
thread_local char g_err[512] = "";
}

void set_error(const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
}

int num_sms() {
    static int n = 0;
    if (n == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 152;
    }
    return n;
}

namespace {

// ---- node <-> unknown maps (CPUSolver.cpp:13-37) --------------------------------
// Stores a state value; a store that changes its bits clears *prev_valid (the
// extrapolated initial guess needs the state the loop itself produced, so a
// field written back unchanged between frames keeps the history).
template <typename R>
__device__ __forceinline__ void store_state(R* dst, R val, int* prev_valid) {
    if (prev_valid) {
        const R old = *dst;
        bool same;
        if constexpr (sizeof(R) == 8) same = __double_as_longlong(old) == __double_as_longlong(val);
        else same = __float_as_uint(old) == __float_as_uint(val);
        if (!same) *prev_valid = 0;
    }
    *dst = val;
}

template <typename R>
__global__ void k_gather_nodes(const float* __restrict__ vals, const int32_t* __restrict__ idx, int64_t V, R* out,
                               int stride, int off, int* prev_valid) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < V; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t k = idx[i];
        if (k >= 0) store_state(out + (int64_t)k * stride + off, (R)vals[i], prev_valid);
    }
}

template <typename R>
__global__ void k_scatter_nodes(const R* __restrict__ in, const int32_t* __restrict__ idx, int64_t V, float* out,
                                int stride, int off) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < V; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t k = idx[i];
        out[i] = k >= 0 ? (float)in[(int64_t)k * stride + off] : 0.0f;
    }
}

template <typename R>
__global__ void k_interleave(const R* __restrict__ u, const R* __restrict__ v, int64_t N, R* uv) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < N; i += (int64_t)gridDim.x * blockDim.x) {
        uv[2 * i] = u[i];
        uv[2 * i + 1] = v[i];
    }
}

template <typename R>
__global__ void k_deinterleave(const R* __restrict__ uv, int64_t N, R* u, R* v) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < N; i += (int64_t)gridDim.x * blockDim.x) {
        u[i] = uv[2 * i];
        v[i] = uv[2 * i + 1];
    }
}

// Caller-order unknown u <-> solver-order index pos[u].
template <typename R>
__global__ void k_copy_to_state(const R* __restrict__ in, const int32_t* __restrict__ pos, int64_t N, R* out,
                                int stride, int off, int* prev_valid) {
    for (int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; u < N; u += (int64_t)gridDim.x * blockDim.x)
        store_state(out + (int64_t)pos[u] * stride + off, in[u], prev_valid);
}

template <typename R>
__global__ void k_copy_from_state(const R* __restrict__ in, const int32_t* __restrict__ pos, int64_t N, R* out,
                                  int stride, int off) {
    for (int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; u < N; u += (int64_t)gridDim.x * blockDim.x)
        out[u] = in[(int64_t)pos[u] * stride + off];
}

__global__ void k_compose_idx(const int32_t* __restrict__ idx, const int32_t* __restrict__ pos, int64_t V,
                              int32_t* idx_c) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < V; i += (int64_t)gridDim.x * blockDim.x)
        idx_c[i] = idx[i] >= 0 ? pos[idx[i]] : -1;
}

// *found = 1 when an unknown has no mass: no triangle, or none with an area.
__global__ void k_bare_rows(int64_t N, const int32_t* __restrict__ diag, const double* __restrict__ M, int* found) {
    for (int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; u < N; u += (int64_t)gridDim.x * blockDim.x)
        if (diag[u] < 0 || !(M[diag[u]] > 0)) *found = 1;
}

template <typename R>
__global__ void k_float_to(const float* __restrict__ in, int64_t n, R* out) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = (R)in[i];
}

// Reads n 16-byte words (evicting the L2 with clean lines); the sink is
// written only for an all-ones word, which the buffer (zeroed) never holds.
__global__ void k_read_flush(const uint4* __restrict__ p, int64_t n, unsigned int* sink) {
    unsigned int acc = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const uint4 v = __ldcg(p + i);
        acc |= v.x & v.y & v.z & v.w;
    }
    if (acc == 0xffffffffu) *sink = acc;
}

template <typename A, typename B>
__global__ void k_convert(const A* __restrict__ in, int64_t n, B* out) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = (B)in[i];
}

}  // namespace

// Everything that depends on the arithmetic type.
struct Fields {
    int64_t N = 0;
    void* u = nullptr;   // R[N]
    void* v = nullptr;   // R[N]
    void* a = nullptr;   // R[N]  Newmark acceleration
    void* ut = nullptr;  // R[N]  Newmark predictors
    void* vt = nullptr;
    void* uv = nullptr;  // R[2N] interleaved (Gray-Scott)
    bool interleaved = false;  // (u, v) currently live in uv
    // solver work, one field (p1 holds the two alternating direction buffers)
    // r1/r2 hold the alternating r, w, s buffers of the Chronopoulos-Gear loop
    void *A1 = nullptr, *d1 = nullptr, *b1 = nullptr, *r1 = nullptr, *z1 = nullptr, *p1 = nullptr, *q1 = nullptr;
    void *A0 = nullptr, *d0 = nullptr;  // Newmark start-up operator (M)
    // two fields
    void *A2 = nullptr, *d2 = nullptr, *b2 = nullptr, *r2 = nullptr, *z2 = nullptr, *p2 = nullptr, *q2 = nullptr;
    void *xprev2 = nullptr, *xg2 = nullptr;  // Gray-Scott: previous state, extrapolated guess
};

// Device buffers a call needs, kept by the handle for the next call of the
// same shape: the k-th request of a call gets the k-th buffer, made anew when
// it is too small.  (Allocating and freeing took 50 us of a frame's normals
// and 0.1 ms a buffer in the adjoints, and each free waits for the device.)
struct Scratch {
    Scratch() = default;
    Scratch(const Scratch&) = delete;
    Scratch& operator=(const Scratch&) = delete;
    ~Scratch() { release(); }
    std::vector<std::pair<void*, size_t>> bufs;
    size_t next = 0;
    void rewind() { next = 0; }
    template <typename T>
    T* alloc(int64_t count) {
        const size_t need = (size_t)(count > 0 ? count : 1) * sizeof(T);
        if (next == bufs.size()) bufs.emplace_back(nullptr, 0);
        auto& b = bufs[next++];
        if (b.second < need) {
            cudaFree(b.first);
            b = {nullptr, 0};
            FEA_CUDA_TRY(cudaMalloc(&b.first, need));
            b.second = need;
        }
        return static_cast<T*>(b.first);
    }
    int64_t bytes() const {
        int64_t n = 0;
        for (const auto& b : bufs) n += (int64_t)b.second;
        return n;
    }
    void release() {
        for (auto& b : bufs) cudaFree(b.first);
        bufs.clear();
        next = 0;
    }
};

// The states of an adjoint sweep: one field per checkpoint and per step of a
// segment, a count the caller chooses.  They go back to the device after a
// sweep that needed more than kStatesKept; below that the handle keeps them
// (freeing and allocating them cost 0.1 ms a buffer and a wait for the device).
constexpr int64_t kStatesKept = (int64_t)64 << 20;
struct SweepStates {
    Scratch& mem;
    explicit SweepStates(Scratch& m) : mem(m) { mem.rewind(); }
    ~SweepStates() {
        if (mem.bytes() > kStatesKept) mem.release();
    }
};

}  // namespace fea

using namespace fea;

struct fea_solver {
    int device = 0;
    cudaStream_t stream = nullptr;
    int precision = FEA_FP32;
    int bc = FEA_DIRICHLET;
    int64_t V = 0, T = 0, nb = 0, N = 0;
    fea_params prm{};
    // mesh
    DeviceArena mesh_mem;
    float* xyz = nullptr;
    uint32_t* tri = nullptr;
    uint8_t* ob = nullptr;
    float* elem_D = nullptr;    // [T] per-element diffusivity (null: 1)
    float* elem_vel = nullptr;  // [3T]
    double* elem_Dr = nullptr;  // diffusivity widened to FP64 for assembly
    // FEMContext state (rebuilt on BC change)
    DeviceArena mat_mem;
    int32_t* idx = nullptr;
    Pattern P;
    double *Kloc = nullptr, *Mloc = nullptr, *Aloc = nullptr;  // element blocks [9T], FP64
    double *K64 = nullptr, *M64 = nullptr, *Adv64 = nullptr;   // assembled in FP64
    void *K = nullptr, *M = nullptr, *Adv = nullptr;           // in the handle's type (export)
    // the solver's ordering of the unknowns (Morton order of their points)
    Pattern Pc;                     // pattern in solver order
    int32_t* pos = nullptr;         // [N] unknown -> solver index
    int32_t* inv = nullptr;         // [N] solver index -> unknown
    int32_t* emap = nullptr;        // [nnz] solver slot -> assembly slot
    int32_t* idx_c = nullptr;       // [V] node -> solver index (-1 on Dirichlet points)
    void *Kc = nullptr, *Mc = nullptr, *Advc = nullptr;        // values in solver order
    TileEll ell;                    // the CG kernels' layout of Pc (tile_ell.cu)
    int stream_stages = 0;          // stages of the streamed iteration that fit in shared memory (0, 2 or 3)
    void *S1 = nullptr, *S0 = nullptr, *S2 = nullptr;          // tile-ELL copies of A1, A0, A2
    void* Ms_ell = nullptr;                                    // tile-ELL copy of M
    TileEll ell_od;                                            // the layout without diagonal entries (ring kernels)
    void *S1d = nullptr, *S0d = nullptr, *S2d = nullptr;       // its copies of A1, A0, A2
    StiffGroups grp;                // groups tied by nearly degenerate triangles (stiff.cu)
    TileEll ell_st;                 // the diagonal-free layout of A' = Q^T A Q
    void *S1s = nullptr, *S0s = nullptr, *S2s = nullptr;       // its copies of A1', A0', A2'
    StiffBasis B1, B0, B2;          // the bases of A1, A0, A2
    bool stiff_stale[3] = {true, true, true};                  // A0', A1', A2' do not match their operators
    void* grp_x0 = nullptr;         // the groups' start values during a solve
    int* grp_in = nullptr;
    bool diagonal_only = false;     // solves without the stiff groups, on the step graph (DiagonalOnly)
    void *Ks_ell = nullptr, *Advs_ell = nullptr;               // tile-ELL copies of K and Adv (resident launches)
    int64_t run_steps = 0;          // steps asked of the last resident run
    bool many_runs = false, later_run = false;  // a call of several runs, past its first (CallRuns)
    int bare = -1;                  // unknowns without mass (bare_rows): -1 not asked
    bool resident = true;           // the step loop may run as one resident launch (no CG variant chosen)
    struct {
        int known = 0;              // 0: not asked, 1: fits, -1: does not
        ResidentPlan plan;
    } res[2][2];                    // by fields - 1 and stiff groups
    void* exchange[2] = {nullptr, nullptr};  // by fields - 1: the blocks' exchange (first resident launch)
    uint8_t* adv_present = nullptr;
    Fields F;
    // loop state
    DeviceArena run_mem;
    StepParams* d_prm = nullptr;
    CgState* d_cg = nullptr;
    RunState* d_run = nullptr;
    double* d_part = nullptr;
    unsigned int* d_tickets = nullptr;
    LoopFlags* d_flags = nullptr;
    bool stream_mode = false;  // FEA_LAUNCH_MODE=stream: kernel-by-kernel launches
    RunState* h_run = nullptr;  // pinned
    StepGraph graph, init_graph;
    StepGraph diag_graph;  // the step graph without the stiff groups
    StepGraph given_graph[2];  // the adjoint's solve by fields - 1, and what it was built for
    struct {
        const void *x = nullptr, *rhs = nullptr, *op = nullptr;
    } given_for[2];
    Scratch scratch[4];  // adjoint sweeps, their entry points, smooth normals, the sweeps' states
    int lanes = 8;  // CG kernel variant: 0/1 tile-ELL (8/4 entries prefetched), 2/3 streamed (stages), 4/8/16 CSR window
    bool op_dirty = true;
    int op_kind = -1;
    bool acc_valid = false;
    float cur_vel[3] = {1.f, 0.f, 0.f};
    int cur_vel_mode = 0;
    float* d_nodes = nullptr;  // node-indexed staging buffer [V] for host field copies
    int32_t* vt_ptr = nullptr;  // vertex -> triangles (built on first use)
    int32_t* vt_tri = nullptr;
};

namespace fea {
namespace {

size_t rsize(const fea_solver* s) { return s->precision == FEA_FP64 ? 8 : 4; }

// Whether a ring variant's iteration fits a block's shared memory on the layout
// L at `stages` stages (both field counts do when two fields do).
bool ring_fits(const fea_solver* s, const TileEll& L, int stages) {
    const size_t need = s->precision == FEA_FP64 ? ring_smem_bytes<double, 2>(L.emax, L.hmax, stages)
                                                 : ring_smem_bytes<float, 2>(L.emax, L.hmax, stages);
    return need <= kStreamSmemLimit;
}
int ring_stages(int lanes) { return lanes == 14 ? 3 : lanes == 15 ? 4 : 0; }

// Tiles per SM up to which a mesh may run as a resident launch (resident.cu
// has kernels for that many).
int64_t resident_tiles(const fea_solver* s) { return s->precision == FEA_FP32 ? 10 : 8; }

int64_t pad_tiles(int64_t n) { return ceil_div(n, kTileRows) * kTileRows; }

void* ralloc(DeviceArena& ar, const fea_solver* s, int64_t n) {
    if (s->precision == FEA_FP64) return ar.alloc<double>(n);
    return ar.alloc<float>(n);
}

// n values of the handle's type past p.
void* roffset(const fea_solver* s, void* p, int64_t n) { return (char*)p + rsize(s) * (size_t)n; }

int step_kind(const fea_params& p) {
    switch (p.equation) {
    case FEA_HEAT: return EQ_HEAT;
    case FEA_ADVECTION_DIFFUSION: return p.advection_scheme == 1 ? EQ_ADV_EXPLICIT : EQ_HEAT;
    case FEA_WAVE: return p.wave_scheme == 1 ? EQ_WAVE_NEWMARK : EQ_WAVE_REF;
    case FEA_REACTION_DIFFUSION: return p.reaction_mode == 1 ? EQ_GS_CONSISTENT : EQ_GS_REF;
    default: return -1;
    }
}

bool two_fields(int kind) { return kind == EQ_GS_REF || kind == EQ_GS_CONSISTENT; }

double time_step(const fea_params& p) {
    switch (p.equation) {
    case FEA_HEAT: return p.heat_time_step;
    case FEA_ADVECTION_DIFFUSION: return p.advdiff_time_step;
    case FEA_WAVE: return p.wave_time_step;
    default: return p.rd_time_step;
    }
}

// Assembly runs in FP64 for both precisions (once per mesh or parameter
// change); FP32 handles then round the assembled values once, so their
// matrices carry only the final FP32 rounding.
void assemble(fea_solver* s) {
    const bool vel_elem = s->prm.velocity_mode == 1 && s->elem_vel;
    element_matrices<double>(s->xyz, s->tri, s->T, vel_elem ? 1 : 0, s->prm.advdiff_velocity, s->elem_vel,
                             s->Kloc, s->Mloc, s->Aloc, s->stream);
    ordered_sum<double>(s->P, s->Kloc, s->elem_Dr, s->K64, s->stream);
    ordered_sum<double>(s->P, s->Mloc, nullptr, s->M64, s->stream);
    ordered_sum_adv<double>(s->P, s->Aloc, s->tri, s->ob, s->Adv64, s->adv_present, s->stream);
    if (s->precision == FEA_FP32) {
        round_copy<float>(s->K64, nullptr, s->P.nnz, (float*)s->K, s->stream);
        round_copy<float>(s->M64, nullptr, s->P.nnz, (float*)s->M, s->stream);
        round_copy<float>(s->Adv64, nullptr, s->P.nnz, (float*)s->Adv, s->stream);
        round_copy<float>(s->K64, s->emap, s->P.nnz, (float*)s->Kc, s->stream);
        round_copy<float>(s->M64, s->emap, s->P.nnz, (float*)s->Mc, s->stream);
        round_copy<float>(s->Adv64, s->emap, s->P.nnz, (float*)s->Advc, s->stream);
        fill_tile_ell<float, 1>(s->ell, (const FV<float, 1>*)s->Mc, (FV<float, 1>*)s->Ms_ell, s->stream);
        if (s->Ks_ell) {
            fill_tile_ell<float, 1>(s->ell, (const FV<float, 1>*)s->Kc, (FV<float, 1>*)s->Ks_ell, s->stream);
            fill_tile_ell<float, 1>(s->ell, (const FV<float, 1>*)s->Advc, (FV<float, 1>*)s->Advs_ell, s->stream);
        }
    } else {
        round_copy<double>(s->K64, s->emap, s->P.nnz, (double*)s->Kc, s->stream);
        round_copy<double>(s->M64, s->emap, s->P.nnz, (double*)s->Mc, s->stream);
        round_copy<double>(s->Adv64, s->emap, s->P.nnz, (double*)s->Advc, s->stream);
        fill_tile_ell<double, 1>(s->ell, (const FV<double, 1>*)s->Mc, (FV<double, 1>*)s->Ms_ell, s->stream);
        if (s->Ks_ell) {
            fill_tile_ell<double, 1>(s->ell, (const FV<double, 1>*)s->Kc, (FV<double, 1>*)s->Ks_ell, s->stream);
            fill_tile_ell<double, 1>(s->ell, (const FV<double, 1>*)s->Advc, (FV<double, 1>*)s->Advs_ell, s->stream);
        }
    }
    memcpy(s->cur_vel, s->prm.advdiff_velocity, sizeof(s->cur_vel));
    s->cur_vel_mode = s->prm.velocity_mode;
    s->op_dirty = true;
}

// The solver's ordering (ordering.cu) and the pattern in it.
void build_ordering(fea_solver* s) {
    cudaStream_t st = s->stream;
    const int64_t V = s->V, N = s->N;
    s->pos = s->mat_mem.alloc<int32_t>(N);
    s->inv = s->mat_mem.alloc<int32_t>(N);
    s->emap = s->mat_mem.alloc<int32_t>(s->P.nnz);
    s->idx_c = s->mat_mem.alloc<int32_t>(V);
    solver_order(s->xyz, s->idx, V, s->P.row_ptr, N, s->inv, s->pos, st);
    k_compose_idx<<<launch_grid(V), kBlock, 0, st>>>(s->idx, s->pos, V, s->idx_c);
    FEA_CHECK_LAUNCH();
    build_permuted(s->P, s->pos, s->inv, s->Pc, s->emap, s->mat_mem, st);
}

// The stiff groups of the mesh and the diagonal-free layout in their basis:
// A' has the pattern of A with the groups' rows and columns filled in.
// False, and no groups, when there are none or the layout does not fit.
bool build_stiff_layout(fea_solver* s) {
    cudaStream_t st = s->stream;
    const int64_t N = s->N;
    if (!stiff_groups_wanted(N)) return false;
    // the groups follow the mesh alone: K without the per-element diffusivity
    element_matrices<double>(s->xyz, s->tri, s->T, 0, s->prm.advdiff_velocity, nullptr, s->Kloc, s->Mloc, s->Aloc, st);
    ordered_sum<double>(s->P, s->Kloc, nullptr, s->K64, st);
    const std::vector<std::array<int32_t, 4>> groups = find_stiff_groups(s->P, s->K64, st);
    StiffGroups G;
    ModRows mod;
    if (groups.empty() || !plan_stiff_rows(groups, s->Pc, s->pos, G, mod, s->mat_mem, st) ||
        !build_tile_ell(s->Pc.row_ptr, s->Pc.col, N, 2 * rsize(s), kEllSmemBudget, s->ell_st, s->mat_mem, st, true,
                        &mod) ||
        !ring_fits(s, s->ell_st, 3)) {  // the groups' rows are longer: the kernel stays, they go
        s->ell_st = TileEll{};
        return false;
    }
    s->grp = G;
    s->S1s = ralloc(s->mat_mem, s, 4 * s->ell_st.E);
    s->S0s = roffset(s, s->S1s, s->ell_st.E);
    s->S2s = roffset(s, s->S0s, s->ell_st.E);
    const std::pair<StiffBasis*, int> bases[3] = {{&s->B1, 1}, {&s->B0, 1}, {&s->B2, 2}};
    for (const auto& b : bases) {
        b.first->Q = s->mat_mem.alloc<double>(16 * (int64_t)G.n * b.second);
        b.first->X = ralloc(s->mat_mem, s, (int64_t)G.nx * b.second);
        b.first->dinv = ralloc(s->mat_mem, s, pad_tiles(N) * b.second);
        FEA_CUDA_TRY(cudaMemsetAsync(b.first->dinv, 0, rsize(s) * (size_t)(pad_tiles(N) * b.second), st));
    }
    s->grp_x0 = ralloc(s->mat_mem, s, 8 * (int64_t)G.n);
    s->grp_in = s->mat_mem.alloc<int>(1);
    FEA_CUDA_TRY(cudaMemsetAsync(s->grp_in, 0, sizeof(int), st));
    return true;
}

// FEMContext::update_boundary_conditions + assemble_matrices and the state.
void build_context(fea_solver* s) {
    s->graph.destroy();
    s->init_graph.destroy();
    s->diag_graph.destroy();
    for (auto& g : s->given_graph) g.destroy();
    s->mat_mem.release();
    s->P = Pattern{};
    s->Pc = Pattern{};
    s->ell = TileEll{};
    s->ell_od = TileEll{};
    s->stream_stages = 0;
    s->S1 = s->S0 = s->S2 = nullptr;
    s->S1d = s->S0d = s->S2d = nullptr;
    s->Ms_ell = nullptr;
    s->bare = -1;
    s->grp = StiffGroups{};
    s->ell_st = TileEll{};
    s->Ks_ell = s->Advs_ell = nullptr;
    for (auto& r : s->res) r[0].known = r[1].known = 0;
    s->exchange[0] = s->exchange[1] = nullptr;
    s->S1s = s->S0s = s->S2s = nullptr;
    s->B1 = s->B0 = s->B2 = StiffBasis{};
    s->F = Fields{};
    cudaStream_t st = s->stream;
    s->idx = s->mat_mem.alloc<int32_t>(s->V);
    s->N = build_idx_map(s->ob, s->V, s->bc, s->idx, st);
    build_pattern(s->P, s->mat_mem, s->tri, s->T, s->ob, s->idx, s->bc, s->N, st);
    const int64_t N = s->N, nnz = s->P.nnz, T = s->T;
    build_ordering(s);
    s->Kloc = s->mat_mem.alloc<double>(9 * T);
    s->Mloc = s->mat_mem.alloc<double>(9 * T);
    s->Aloc = s->mat_mem.alloc<double>(9 * T);
    s->K64 = s->mat_mem.alloc<double>(nnz);
    s->M64 = s->mat_mem.alloc<double>(nnz);
    s->Adv64 = s->mat_mem.alloc<double>(nnz);
    {
        const int32_t *rp = s->Pc.row_ptr, *col = s->Pc.col;
        build_tile_ell(rp, col, N, 2 * rsize(s), kEllSmemBudget, s->ell, s->mat_mem, st);
        if (s->ell.ok) {
            // one allocation per layout (E is a multiple of 32 entries)
            const bool extra = ceil_div(N, kTileRows) <= resident_tiles(s) * (int64_t)num_sms();
            s->S1 = ralloc(s->mat_mem, s, (extra ? 7 : 5) * s->ell.E);
            s->S0 = roffset(s, s->S1, s->ell.E);
            s->S2 = roffset(s, s->S0, s->ell.E);
            s->Ms_ell = roffset(s, s->S2, 2 * s->ell.E);
            if (extra) {
                s->Ks_ell = roffset(s, s->Ms_ell, s->ell.E);
                s->Advs_ell = roffset(s, s->Ks_ell, s->ell.E);
            }
            if (build_tile_ell(rp, col, N, 2 * rsize(s), kEllSmemBudget, s->ell_od, s->mat_mem, st, true)) {
                s->S1d = ralloc(s->mat_mem, s, 4 * s->ell_od.E);
                s->S0d = roffset(s, s->S1d, s->ell_od.E);
                s->S2d = roffset(s, s->S0d, s->ell_od.E);
            }
            build_stiff_layout(s);
        }
        // both field counts fit when the two-field stages do
        const size_t stage = s->precision == FEA_FP64 ? stream_stage_bytes<double, 2>(s->ell.emax, s->ell.hmax)
                                                      : stream_stage_bytes<float, 2>(s->ell.emax, s->ell.hmax);
        s->stream_stages = !s->ell.ok ? 0 : 3 * stage <= kStreamSmemLimit ? 3 : 2 * stage <= kStreamSmemLimit ? 2 : 0;
        // default variant: direct row loads with the operator ring (14) when
        // its stages fit, else the streamed deferred-finish kernel with as
        // many stages as fit, else the tile-ELL kernel, else windowed CSR
        s->lanes = !s->ell.ok ? 8
                   : ring_fits(s, s->ell, 3)  ? 14
                   : s->stream_stages >= 3    ? 11
                   : s->stream_stages >= 2    ? 10
                                              : 0;
    }
    if (s->precision == FEA_FP64) {
        s->K = s->K64;
        s->M = s->M64;
        s->Adv = s->Adv64;
    } else {
        s->K = ralloc(s->mat_mem, s, nnz);
        s->M = ralloc(s->mat_mem, s, nnz);
        s->Adv = ralloc(s->mat_mem, s, nnz);
    }
    s->Kc = ralloc(s->mat_mem, s, nnz);
    s->Mc = ralloc(s->mat_mem, s, nnz);
    s->Advc = ralloc(s->mat_mem, s, nnz);
    s->adv_present = s->mat_mem.alloc<uint8_t>(nnz);
    Fields& F = s->F;
    F.N = N;
    // every per-row vector holds whole tiles (Nt rows, zero beyond N): the
    // streamed CG kernels copy 256-row tiles of them into shared memory
    const int64_t Nt = ceil_div(N, kTileRows) * kTileRows;
    F.u = ralloc(s->mat_mem, s, Nt);
    F.v = ralloc(s->mat_mem, s, Nt);
    F.a = ralloc(s->mat_mem, s, Nt);
    F.ut = ralloc(s->mat_mem, s, Nt);
    F.vt = ralloc(s->mat_mem, s, Nt);
    F.uv = ralloc(s->mat_mem, s, 2 * Nt);
    F.A1 = ralloc(s->mat_mem, s, nnz);
    F.d1 = ralloc(s->mat_mem, s, Nt);
    F.b1 = ralloc(s->mat_mem, s, Nt);
    const int64_t Np = Nt;  // every buffer of a group starts on a tile boundary
    F.r1 = ralloc(s->mat_mem, s, 6 * Np);  // r, w, s: two buffers each
    F.z1 = ralloc(s->mat_mem, s, Nt);
    F.p1 = ralloc(s->mat_mem, s, 2 * Np);
    F.q1 = ralloc(s->mat_mem, s, Nt);
    F.A0 = ralloc(s->mat_mem, s, nnz);
    F.d0 = ralloc(s->mat_mem, s, Nt);
    F.A2 = ralloc(s->mat_mem, s, 2 * nnz);
    F.d2 = ralloc(s->mat_mem, s, 2 * Nt);
    F.b2 = ralloc(s->mat_mem, s, 2 * Nt);
    F.r2 = ralloc(s->mat_mem, s, 12 * Np);
    F.z2 = ralloc(s->mat_mem, s, 2 * Nt);
    F.p2 = ralloc(s->mat_mem, s, 4 * Np);
    F.q2 = ralloc(s->mat_mem, s, 2 * Nt);
    F.xprev2 = ralloc(s->mat_mem, s, 2 * Nt);
    F.xg2 = ralloc(s->mat_mem, s, 2 * Nt);
    // every vector starts at zero (the direction buffers are read with weight
    // beta = 0 only after a write, but a zero start keeps them finite)
    const std::pair<void*, int64_t> zeroed[] = {
        {F.u, Nt}, {F.v, Nt}, {F.a, Nt}, {F.ut, Nt}, {F.vt, Nt}, {F.uv, 2 * Nt}, {F.d1, Nt}, {F.b1, Nt},
        {F.r1, 6 * Np}, {F.z1, Nt}, {F.p1, 2 * Np}, {F.q1, Nt}, {F.d0, Nt}, {F.d2, 2 * Nt}, {F.b2, 2 * Nt},
        {F.r2, 12 * Np}, {F.z2, 2 * Nt}, {F.p2, 4 * Np}, {F.q2, 2 * Nt}, {F.xprev2, 2 * Nt}, {F.xg2, 2 * Nt}};
    for (const auto& zv : zeroed)
        FEA_CUDA_TRY(cudaMemsetAsync(zv.first, 0, rsize(s) * (size_t)(zv.second > 0 ? zv.second : 1), st));
    F.interleaved = false;
    s->acc_valid = false;
    assemble(s);
    FEA_CUDA_TRY(cudaStreamSynchronize(st));
}

// The FP32 wave on larger meshes keeps the diagonal iteration on the step graph,
// bit for bit: its velocity sums accelerations -c^2 M^-1 K u whose FP32 rounding
// grows with the mesh, and another order of the sums moves it by a large part of
// that error.  Ten Newmark steps, four starts, velocity against 64 bits with this
// rule and without it (groups; the resident launch where it fits), and how far the two are apart:
// grid 200 x 200 3.1 to 6.1e-5 either way, apart 0.9 to 1.7e-5; 500 x 500 7.0e-5 to
// 1.7e-4 against 6.7e-5 to 1.6e-4, apart 4.5 to 8.3e-5; 900 x 900 9.1e-5 to 2.8e-4
// against 8.7e-5 to 2.3e-4, apart 6.3e-5 to 2.0e-4.  So the rule keeps bits, not
// accuracy; without it those runs take 1.3 ms for 2.6, 2.3 for 10 and 7.5 for 33.
bool rounding_bound_wave(const fea_solver* s) {
    return s->precision == FEA_FP32 && s->prm.equation == FEA_WAVE && s->N > 16384;
}

// Whether some unknown of the mesh has no mass, as a vertex that no triangle
// names (asked once per assembly, by the equation it matters to).
bool bare_rows(fea_solver* s) {
    if (s->bare < 0) {
        DeviceArena tmp;
        int* found = tmp.alloc<int>(1);
        FEA_CUDA_TRY(cudaMemsetAsync(found, 0, sizeof(int), s->stream));
        k_bare_rows<<<launch_grid(s->N), kBlock, 0, s->stream>>>(s->N, s->P.diag, s->M64, found);
        FEA_CHECK_LAUNCH();
        int h = 0;
        FEA_CUDA_TRY(cudaMemcpyAsync(&h, found, sizeof(int), cudaMemcpyDeviceToHost, s->stream));
        FEA_CUDA_TRY(cudaStreamSynchronize(s->stream));
        s->bare = h;
    }
    return s->bare > 0;
}

// The nodal reaction (the reference's) on a mesh with such unknowns: their
// equations read 0 = reaction, the system has no solution, and the step graph's
// diagonal iteration reports it (the value runs away past 1e4, as it does
// under the reference's CG).  Started from the diagonal-free product, as the
// resident launch and the groups do, CG would take the row's diagonal for 1 and
// converge on a value that solves nothing.  Under every other equation such a row's
// right-hand side is 0.
bool nodal_on_bare_rows(fea_solver* s) { return step_kind(s->prm) == EQ_GS_REF && bare_rows(s); }

// Whether variant l iterates in the basis of the handle's stiff groups.
bool stiff_variant(const fea_solver* s, int l) {
    return s->grp.n > 0 && is_ring_variant(l) && ring_fits(s, s->ell_st, ring_stages(l));
}

// Whether the current equation's solves run in the stiff groups' basis.
// Implicit advection-diffusion does not: its operator is not symmetric, CG
// may break down on it, and it keeps the iteration it had.
bool stiff_solves(fea_solver* s) {
    if (rounding_bound_wave(s)) return false;
    const bool symmetric = s->prm.equation != FEA_ADVECTION_DIFFUSION || s->prm.advection_scheme == 1;
    return stiff_variant(s, s->lanes) && !s->diagonal_only && symmetric && !nodal_on_bare_rows(s);
}

// r, w and s of the Chronopoulos-Gear iteration, two buffers each, carved
// from one allocation of 6 * Np unknowns.
template <typename R, int NF>
void set_rws(StepArgs<R, NF>& a, FV<R, NF>* base, int64_t Np) {
    for (int k = 0; k < 2; k++) {
        a.rb[k] = base + k * Np;
        a.wb[k] = base + (2 + k) * Np;
        a.sb[k] = base + (4 + k) * Np;
    }
}

// The copy of A' = Q^T A Q in the stiff groups' basis, made when a solve first
// wants it after the operator changed.
template <typename R, int NF>
void ensure_stiff(fea_solver* s, bool init_op) {
    bool& stale = s->stiff_stale[NF == 2 ? 2 : init_op ? 0 : 1];
    if (!stale) return;
    const Fields& F = s->F;
    const auto* A = (const FV<R, NF>*)(NF == 2 ? F.A2 : init_op ? F.A0 : F.A1);
    const auto* dinv = (const FV<R, NF>*)(NF == 2 ? F.d2 : init_op ? F.d0 : F.d1);
    const StiffBasis& B = NF == 2 ? s->B2 : init_op ? s->B0 : s->B1;
    void* Ss = NF == 2 ? s->S2s : init_op ? s->S0s : s->S1s;
    update_stiff_basis<R, NF>(s->grp, s->Pc, A, dinv, B, s->stream);
    fill_tile_ell<R, NF>(s->ell_st, A, (FV<R, NF>*)Ss, s->stream, (const FV<R, NF>*)B.X, s->P.nnz);
    stale = false;
}

template <typename R, int NF>
StepArgs<R, NF> make_args(fea_solver* s, bool init_op) {
    StepArgs<R, NF> a{};
    Fields& F = s->F;
    a.N = (int)s->N;
    a.rp = s->Pc.row_ptr;
    a.col = s->Pc.col;
    a.M = (const R*)s->Mc;
    a.K = (const R*)s->Kc;
    a.Adv = (const R*)s->Advc;
    if constexpr (NF == 1) {
        a.A = (const FV<R, 1>*)(init_op ? F.A0 : F.A1);
        a.dinv = (const FV<R, 1>*)(init_op ? F.d0 : F.d1);
        a.b = (FV<R, 1>*)F.b1;
        set_rws(a, (FV<R, 1>*)F.r1, pad_tiles(s->N));
        a.z = (FV<R, 1>*)F.z1;
        a.pp[0] = (FV<R, 1>*)F.p1;
        a.pp[1] = a.pp[0] + pad_tiles(s->N);
        a.q = (FV<R, 1>*)F.q1;
    } else {
        a.A = (const FV<R, 2>*)F.A2;
        a.dinv = (const FV<R, 2>*)F.d2;
        a.b = (FV<R, 2>*)F.b2;
        set_rws(a, (FV<R, 2>*)F.r2, pad_tiles(s->N));
        a.z = (FV<R, 2>*)F.z2;
        a.pp[0] = (FV<R, 2>*)F.p2;
        a.pp[1] = a.pp[0] + pad_tiles(s->N);
        a.q = (FV<R, 2>*)F.q2;
    }
    a.u = (R*)F.u;
    a.v = (R*)F.v;
    a.a = (R*)F.a;
    a.ut = (R*)F.ut;
    a.vt = (R*)F.vt;
    if (s->ell.ok) {
        if constexpr (NF == 1) a.As = (const FV<R, 1>*)(init_op ? s->S0 : s->S1);
        else a.As = (const FV<R, 2>*)s->S2;
        a.lcol = s->ell.lcol;
        a.lcol2 = s->ell.lcol2;
        a.slice_off = s->ell.slice_off;
        a.halo_off = s->ell.halo_off;
        a.halo_col = s->ell.halo_col;
        a.hmax = s->ell.hmax;
        a.emax = s->ell.emax;
        a.Ms = (const R*)s->Ms_ell;
        const bool stiff = stiff_solves(s);
        const TileEll& od = stiff ? s->ell_st : s->ell_od;
        if (od.ok) {
            if constexpr (NF == 1)
                a.As_od = (const FV<R, 1>*)(stiff ? (init_op ? s->S0s : s->S1s) : (init_op ? s->S0d : s->S1d));
            else
                a.As_od = (const FV<R, 2>*)(stiff ? s->S2s : s->S2d);
            a.lcol_od = od.lcol;
            a.slice_off_od = od.slice_off;
            a.halo_off_od = od.halo_off;
            a.halo_col_od = od.halo_col;
            a.hmax_od = od.hmax;
            a.emax_od = od.emax;
        }
        if (stiff) {
            ensure_stiff<R, NF>(s, init_op);
            const StiffBasis& B = NF == 2 ? s->B2 : init_op ? s->B0 : s->B1;
            a.dinv_it = (const FV<R, NF>*)B.dinv;
            a.ngrp = s->grp.n;
            a.grp_mem = s->grp.mem;
            a.grp_Q = B.Q;
            a.grp_x0 = (FV<R, NF>*)s->grp_x0;
            a.grp_in = s->grp_in;
        }
    }
    if (!a.dinv_it) a.dinv_it = a.dinv;
    a.prm = s->d_prm;
    a.cg = s->d_cg + 1;
    a.cg_alt = s->d_cg;
    a.defer = is_deferred_variant(s->lanes) ? 1 : 0;
    a.run = s->d_run;
    a.part = s->d_part;
    a.part_stride = max_grid_blocks();
    a.tickets = s->d_tickets;
    return a;
}

// Unknown vector of the solve for each kind.
template <typename R, int NF>
void set_x(fea_solver* s, StepArgs<R, NF>& a, int kind) {
    Fields& F = s->F;
    if constexpr (NF == 2) {
        a.x = (FV<R, 2>*)F.uv;
        if (kind == EQ_GS_REF || kind == EQ_GS_CONSISTENT) {  // the initial-guess extrapolation's buffers
            a.xprev = (FV<R, 2>*)F.xprev2;
            a.xg = (FV<R, 2>*)F.xg2;
        }
    } else {
        if (kind == EQ_WAVE_REF) a.x = (FV<R, 1>*)F.v;
        else if (kind == EQ_WAVE_NEWMARK || kind == EQ_NEWMARK_INIT) a.x = (FV<R, 1>*)F.a;
        else a.x = (FV<R, 1>*)F.u;
    }
}

template <typename R>
void upload_params(fea_solver* s) {
    const fea_params& p = s->prm;
    StepParams h{};
    h.dt = time_step(p);
    h.F = p.rd_feed_rate;
    h.k = p.rd_kill_rate;
    const R c = (R)p.wave_c;
    h.c2 = (double)(R)(c * c);
    h.beta = p.newmark_beta;
    h.gamma = p.newmark_gamma;
    h.adv_sign = p.advection_sign;
    FEA_CUDA_TRY(cudaMemcpyAsync(s->d_prm, &h, sizeof(h), cudaMemcpyHostToDevice, s->stream));
    RunState r{};
    FEA_CUDA_TRY(cudaMemcpyAsync(&r, s->d_run, sizeof(r), cudaMemcpyDeviceToHost, s->stream));
    FEA_CUDA_TRY(cudaStreamSynchronize(s->stream));
    double tol = p.cg_tolerance;
    if (!(tol > 0.0)) tol = s->precision == FEA_FP64 ? 1e-10 : 1.1920928955078125e-07;
    r.tol = tol;
    r.max_iter = p.cg_max_iterations > 0 ? p.cg_max_iterations : (int)(2 * s->N > 0x7fffffff ? 0x7fffffff : 2 * s->N);
    r.refine = p.cg_refine;
    if (r.guess != p.cg_initial_guess) r.prev_valid = 0;  // a new rule starts from the warm start
    r.guess = p.cg_initial_guess;
    FEA_CUDA_TRY(cudaMemcpyAsync(s->d_run, &r, sizeof(r), cudaMemcpyHostToDevice, s->stream));
    FEA_CUDA_TRY(cudaStreamSynchronize(s->stream));
}

// Operator coefficients (the float parameters widened to double; the
// operator is evaluated in FP64 and rounded once to the handle's type).
template <typename R>
void update_operator(fea_solver* s, int kind) {
    const fea_params& p = s->prm;
    for (bool& stale : s->stiff_stale) stale = true;
    const double dt = time_step(p);
    if (kind == EQ_GS_REF || kind == EQ_GS_CONSISTENT) {
        OpCoef<2> c{};
        c.f[0] = {dt, (double)p.rd_Du, 1.0, 0.0};
        c.f[1] = {dt, (double)p.rd_Dv, 1.0, 0.0};
        combine_operator<R, 2>(s->Pc, s->emap, s->M64, s->K64, s->Adv64, c, (FV<R, 2>*)s->F.A2, (FV<R, 2>*)s->F.d2,
                               s->stream);
        fill_tile_ell<R, 2>(s->ell, (const FV<R, 2>*)s->F.A2, (FV<R, 2>*)s->S2, s->stream);
        fill_tile_ell<R, 2>(s->ell_od, (const FV<R, 2>*)s->F.A2, (FV<R, 2>*)s->S2d, s->stream);
    } else {
        OpCoef<1> c{};
        c.f[0] = {dt, 0.0, 1.0, 0.0};
        if (kind == EQ_HEAT && p.equation == FEA_HEAT) {
            c.f[0].k1 = p.heat_conductivity;
        } else if (kind == EQ_HEAT) {  // implicit advection-diffusion, CPUSolver.cpp:95
            c.f[0].k1 = p.advdiff_c;
            c.f[0].a1 = -1.0;
        } else if (kind == EQ_ADV_EXPLICIT) {
            c.f[0].k1 = p.advdiff_c;
        } else if (kind == EQ_WAVE_REF) {  // M/dt + (c^2 K) dt, CPUSolver.cpp:113
            const double cc = p.wave_c;
            c.f[0].k1 = cc * cc;
            c.f[0].k2 = dt;
        } else {  // Newmark: M + (beta dt^2 c^2) K
            const double cc = p.wave_c;
            c.f[0].md = 1.0;
            c.f[0].k1 = p.newmark_beta * dt * dt * (cc * cc);
            OpCoef<1> m{};
            m.f[0] = {1.0, 0.0, 1.0, 0.0};
            combine_operator<R, 1>(s->Pc, s->emap, s->M64, s->K64, s->Adv64, m, (FV<R, 1>*)s->F.A0, (FV<R, 1>*)s->F.d0,
                                   s->stream);
            fill_tile_ell<R, 1>(s->ell, (const FV<R, 1>*)s->F.A0, (FV<R, 1>*)s->S0, s->stream);
            fill_tile_ell<R, 1>(s->ell_od, (const FV<R, 1>*)s->F.A0, (FV<R, 1>*)s->S0d, s->stream);
        }
        combine_operator<R, 1>(s->Pc, s->emap, s->M64, s->K64, s->Adv64, c, (FV<R, 1>*)s->F.A1, (FV<R, 1>*)s->F.d1,
                               s->stream);
        fill_tile_ell<R, 1>(s->ell, (const FV<R, 1>*)s->F.A1, (FV<R, 1>*)s->S1, s->stream);
        fill_tile_ell<R, 1>(s->ell_od, (const FV<R, 1>*)s->F.A1, (FV<R, 1>*)s->S1d, s->stream);
    }
}

// Fields changed from outside the step loop: the next step starts its solves
// from the previous solution (the initial-guess extrapolation needs two steps
// of the loop's own history).
void invalidate_guess(fea_solver* s) {
    if (s->d_run) FEA_CUDA_TRY(cudaMemsetAsync(&s->d_run->prev_valid, 0, sizeof(int), s->stream));
}

// Forces the previous-solution start while it lives (the adjoints recompute
// forward states from checkpoints and must reproduce them exactly), then
// restores the handle's rule.
struct GuessOff {
    fea_solver* s;
    explicit GuessOff(fea_solver* h) : s(h) {
        const int zero = 0;
        FEA_CUDA_TRY(cudaMemcpyAsync(&s->d_run->guess, &zero, sizeof(int), cudaMemcpyHostToDevice, s->stream));
        FEA_CUDA_TRY(cudaStreamSynchronize(s->stream));
    }
    ~GuessOff() {
        const int g = s->prm.cg_initial_guess;
        cudaMemcpyAsync(&s->d_run->guess, &g, sizeof(int), cudaMemcpyHostToDevice, s->stream);
        cudaMemsetAsync(&s->d_run->prev_valid, 0, sizeof(int), s->stream);
        cudaStreamSynchronize(s->stream);
    }
};

// Solves without the stiff groups and on the step graph while it lives: the FP32
// Gray-Scott adjoint keeps the bits of the iteration it was validated with, its
// FP64 parameter gradients included.  Against 64 bits, four starts, with this and
// without it: loss on the 400 x 400 grid 0.3 to 4.1e-7 against 4.3 to 6.0e-7, on 512
// x 512 3.8e-7 to 1.2e-6 against 2.9 to 9.4e-7; dJ/du0 4.6 to 5.8e-6 against 4.0 to
// 4.4e-6, and 5.9 to 9.1e-6 against 7.7 to 8.3e-6; the four rates 0.9 to 8.7e-7 against
// 2.3 to 7.4e-7, and 3.4e-7 to 2.3e-6 against 2.2e-7 to 2.6e-6.  Neither is the more
// accurate throughout; without it a 512 x 512 sweep takes 22 ms for 53.
struct DiagonalOnly {
    fea_solver* s;
    DiagonalOnly(fea_solver* h, bool on) : s(h) { s->diagonal_only = on; }
    ~DiagonalOnly() { s->diagonal_only = false; }
};

template <typename R>
void ensure_layout(fea_solver* s, bool interleaved) {
    Fields& F = s->F;
    if (F.interleaved == interleaved || F.N == 0) {
        F.interleaved = interleaved;
        return;
    }
    if (interleaved)
        k_interleave<R><<<launch_grid(F.N), kBlock, 0, s->stream>>>((R*)F.u, (R*)F.v, F.N, (R*)F.uv);
    else
        k_deinterleave<R><<<launch_grid(F.N), kBlock, 0, s->stream>>>((R*)F.uv, F.N, (R*)F.u, (R*)F.v);
    FEA_CHECK_LAUNCH();
    invalidate_guess(s);
    F.interleaved = interleaved;
}

// The flags of the last run go as another starts.  A call of several runs
// (Newmark's starting acceleration and its steps, an adjoint's solves) keeps
// word of an expired wait through all of them (CallRuns).
void clear_run_flags(fea_solver* s) {
    FEA_CUDA_TRY(cudaMemsetAsync(&s->d_run->flags, 0, s->later_run ? kRunFlagBytes : kCallFlagBytes, s->stream));
    if (s->many_runs) s->later_run = true;
}
struct CallRuns {
    fea_solver* s;
    bool outer;  // (the adjoints' calls hold the steps' calls)
    explicit CallRuns(fea_solver* h) : s(h), outer(!h->many_runs) {
        if (outer) s->later_run = false;
        s->many_runs = true;
    }
    ~CallRuns() {
        if (outer) s->many_runs = s->later_run = false;
    }
};
// The loss of a sweep, once no wait of its solves expired.
double sweep_result(fea_solver* s, const double* J) {
    double h = 0;
    int expired = 0;
    FEA_CUDA_TRY(cudaMemcpyAsync(&h, J, sizeof(double), cudaMemcpyDeviceToHost, s->stream));
    FEA_CUDA_TRY(cudaMemcpyAsync(&expired, &s->d_run->expired, sizeof(int), cudaMemcpyDeviceToHost, s->stream));
    FEA_CUDA_TRY(cudaStreamSynchronize(s->stream));
    if (expired) {
        set_error("a wait between the blocks of a solve expired");
        throw Error{FEA_ERR_SOLVE};
    }
    return h;
}

// The resident launch's shape for these arguments, or null: the step graph.
template <typename R, int NF>
const ResidentPlan* resident_plan(fea_solver* s, const StepArgs<R, NF>& a) {
    if (!s->resident || s->stream_mode || s->diagonal_only || !s->Ks_ell || rounding_bound_wave(s) ||
        nodal_on_bare_rows(s))
        return nullptr;
    auto& r = s->res[NF - 1][a.ngrp ? 1 : 0];
    if (r.known == 0) r.known = plan_resident<R, NF>(a, r.plan) ? 1 : -1;
    return r.known > 0 ? &r.plan : nullptr;
}

template <typename R, int NF>
bool try_resident(fea_solver* s, const StepArgs<R, NF>& a, int kind, int64_t nsteps) {
    const ResidentPlan* p = resident_plan<R, NF>(s, a);
    if (!p) return false;
    void*& ex = s->exchange[NF - 1];
    if (!ex) {
        const size_t n = resident_exchange_bytes<R, NF>(s->N);
        ex = s->mat_mem.alloc<unsigned char>((int64_t)n);
        FEA_CUDA_TRY(cudaMemsetAsync(ex, 0, n, s->stream));
    }
    s->run_steps = nsteps;
    clear_run_flags(s);
    run_resident<R, NF>(a, *p, (const R*)s->Ks_ell, (const R*)s->Advs_ell, s->grp.where, ex, kind, nsteps, s->stream);
    return true;
}

template <typename R, int NF>
void run_graph(fea_solver* s, StepGraph& g, int kind, bool init_op, int64_t nsteps) {
    const bool stream_mode = s->stream_mode;
    {
        StepArgs<R, NF> a = make_args<R, NF>(s, init_op);
        set_x<R, NF>(s, a, kind);
        if (try_resident<R, NF>(s, a, kind, nsteps)) return;
    }
    if (!stream_mode && (!g.exec || g.kind != kind || g.lanes != s->lanes)) {
        StepArgs<R, NF> a = make_args<R, NF>(s, init_op);
        set_x<R, NF>(s, a, kind);
        build_step_graph<R, NF>(g, a, kind, s->lanes, s->d_flags);
    }
    long long ctl[2] = {nsteps, 0};  // steps_left, steps_done
    FEA_CUDA_TRY(cudaMemcpyAsync(s->d_run, ctl, sizeof(ctl), cudaMemcpyHostToDevice, s->stream));
    clear_run_flags(s);
    if (stream_mode) {
        StepArgs<R, NF> a = make_args<R, NF>(s, init_op);
        set_x<R, NF>(s, a, kind);
        run_steps_stream<R, NF>(a, kind, s->lanes, s->d_flags, s->stream);
    } else {
        FEA_CUDA_TRY(cudaGraphLaunch(g.exec, s->stream));
    }
}

template <typename R>
void advance(fea_solver* s, int64_t nsteps) {
    const int kind = step_kind(s->prm);
    if (kind < 0) throw Error{FEA_ERR_INVALID_ARGUMENT};
    const bool vel_changed = s->prm.velocity_mode != s->cur_vel_mode ||
                             memcmp(s->cur_vel, s->prm.advdiff_velocity, sizeof(s->cur_vel)) != 0;
    if (vel_changed) assemble(s);
    if (s->op_dirty || s->op_kind != kind) {
        update_operator<R>(s, kind);
        s->op_dirty = false;
        s->op_kind = kind;
    }
    ensure_layout<R>(s, two_fields(kind));
    const CallRuns runs(s);
    if (kind == EQ_WAVE_NEWMARK && !s->acc_valid) {
        // a0 from M a0 = -c^2 K u0
        FEA_CUDA_TRY(cudaMemsetAsync(s->F.a, 0, rsize(s) * (size_t)(s->N > 0 ? s->N : 1), s->stream));
        run_graph<R, 1>(s, s->init_graph, EQ_NEWMARK_INIT, true, 1);
        s->acc_valid = true;
    }
    StepGraph& graph = stiff_solves(s) ? s->graph : s->diag_graph;
    if (two_fields(kind)) run_graph<R, 2>(s, graph, kind, false, nsteps);
    else run_graph<R, 1>(s, graph, kind, false, nsteps);
}

void check_handle(const fea_solver* s) {
    if (!s) {
        set_error("null handle");
        throw Error{FEA_ERR_INVALID_ARGUMENT};
    }
    FEA_CUDA_TRY(cudaSetDevice(s->device));
}

// The device alias of a page-locked host buffer, or nullptr for pageable
// memory.  Page-locked host memory is mapped into the device's address space
// (unified addressing), so the node gather and scatter kernels read and write
// it directly over the host link, in one pass and without the staging copy.
const void* mapped_alias(const void* host) {
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, host) != cudaSuccess) {
        (void)cudaGetLastError();  // an unknown pointer is pageable memory
        return nullptr;
    }
    return at.type == cudaMemoryTypeHost ? at.devicePointer : nullptr;
}

// Host fields travel through the handle's node-sized staging buffer, or are
// read and written in place when the caller's buffer is page-locked.
template <typename R>
void set_node_field(fea_solver* s, const float* host, int which /*0 u, 1 v*/) {
    const float* d = static_cast<const float*>(mapped_alias(host));
    if (!d) {
        FEA_CUDA_TRY(cudaMemcpyAsync(s->d_nodes, host, sizeof(float) * s->V, cudaMemcpyHostToDevice, s->stream));
        d = s->d_nodes;
    }
    Fields& F = s->F;
    int* pv = s->d_run ? &s->d_run->prev_valid : nullptr;
    if (F.interleaved)
        k_gather_nodes<R><<<launch_grid(s->V), kBlock, 0, s->stream>>>(d, s->idx_c, s->V, (R*)F.uv, 2, which, pv);
    else
        k_gather_nodes<R><<<launch_grid(s->V), kBlock, 0, s->stream>>>(d, s->idx_c, s->V,
                                                                        (R*)(which ? F.v : F.u), 1, 0, pv);
    FEA_CHECK_LAUNCH();
    FEA_CUDA_TRY(cudaStreamSynchronize(s->stream));
}

template <typename R>
void get_node_field(fea_solver* s, float* host, int which) {
    float* mapped = static_cast<float*>(const_cast<void*>(mapped_alias(host)));
    float* d = mapped ? mapped : s->d_nodes;
    Fields& F = s->F;
    if (F.interleaved)
        k_scatter_nodes<R><<<launch_grid(s->V), kBlock, 0, s->stream>>>((R*)F.uv, s->idx_c, s->V, d, 2, which);
    else
        k_scatter_nodes<R><<<launch_grid(s->V), kBlock, 0, s->stream>>>((R*)(which ? F.v : F.u), s->idx_c, s->V, d,
                                                                         1, 0);
    FEA_CHECK_LAUNCH();
    if (!mapped)
        FEA_CUDA_TRY(cudaMemcpyAsync(host, d, sizeof(float) * s->V, cudaMemcpyDeviceToHost, s->stream));
    FEA_CUDA_TRY(cudaStreamSynchronize(s->stream));
}

template <typename R>
void copy_field_device(fea_solver* s, const void* src, void* dst, int which, bool to_state) {
    Fields& F = s->F;
    const int64_t N = s->N;
    if (N == 0) return;
    R* state = F.interleaved ? (R*)F.uv : (R*)(which ? F.v : F.u);
    const int st = F.interleaved ? 2 : 1, off = F.interleaved ? which : 0;
    if (to_state) {
        int* pv = s->d_run ? &s->d_run->prev_valid : nullptr;
        k_copy_to_state<R><<<launch_grid(N), kBlock, 0, s->stream>>>((const R*)src, s->pos, N, state, st, off, pv);
    } else
        k_copy_from_state<R><<<launch_grid(N), kBlock, 0, s->stream>>>(state, s->pos, N, (R*)dst, st, off);
    FEA_CHECK_LAUNCH();
}

int displayed_field(const fea_params& p) { return p.equation == FEA_REACTION_DIFFUSION ? 1 : 0; }

// Arguments of the timing probe on the current equation's operator.
template <typename R, int NF>
StepArgs<R, NF> probe_args(fea_solver* s, int kind) {
    StepArgs<R, NF> a = make_args<R, NF>(s, false);
    set_x<R, NF>(s, a, kind);
    a.cont = &s->d_flags->probe;
    a.use_graph = 0;
    a.probe = 1;
    return a;
}

// One probe launch (prepare: mask the fields first, outside any timing).
template <typename R>
void probe(fea_solver* s, int kind, int lanes, bool prepare) {
    if (two_fields(kind)) {
        const StepArgs<R, 2> a = probe_args<R, 2>(s, kind);
        if (prepare) prepare_probe<R, 2>(a, s->stream);
        else launch_spmv_probe<R, 2>(a, lanes, s->stream);
    } else {
        const StepArgs<R, 1> a = probe_args<R, 1>(s, kind);
        if (prepare) prepare_probe<R, 1>(a, s->stream);
        else launch_spmv_probe<R, 1>(a, lanes, s->stream);
    }
}

void probe_any(fea_solver* s, int kind, int lanes, bool prepare) {
    if (s->precision == FEA_FP64) probe<double>(s, kind, lanes, prepare);
    else probe<float>(s, kind, lanes, prepare);
}

// The operator of `kind` up to date (the probe times the current equation).
void ensure_operator(fea_solver* s, int kind) {
    if (s->op_dirty || s->op_kind != kind) {
        if (s->precision == FEA_FP64) update_operator<double>(s, kind);
        else update_operator<float>(s, kind);
        s->op_dirty = false;
        s->op_kind = kind;
    }
}

// ---- adjoint of the explicit advection-diffusion step -------------------------------
// (recurrences in adjoint.cu).  The transposed solves mu = A^-1 lam run the
// forward operator (A is symmetric) through the step graph with a given
// right-hand side; forward states are recomputed from checkpoints taken every
// `ckpt` steps.

// One solve A mu = lam.  The graph is kept for the handle's next sweep; it
// holds the addresses of mu, lam and the operator, and is rebuilt when one
// of them (or the variant) is another.
template <typename R, int NF>
void run_given(fea_solver* s, const StepArgs<R, NF>& a) {
    if (try_resident<R, NF>(s, a, EQ_GIVEN, 1)) return;
    long long ctl[2] = {1, 0};  // steps_left, steps_done
    FEA_CUDA_TRY(cudaMemcpyAsync(s->d_run, ctl, sizeof(ctl), cudaMemcpyHostToDevice, s->stream));
    clear_run_flags(s);
    if (s->stream_mode) {
        run_steps_stream<R, NF>(a, EQ_GIVEN, s->lanes, s->d_flags, s->stream);
        return;
    }
    StepGraph& g = s->given_graph[NF - 1];
    auto& f = s->given_for[NF - 1];
    if (!g.exec || g.lanes != s->lanes || f.x != a.x || f.rhs != a.rhs || f.op != a.As_od) {
        FEA_CUDA_TRY(cudaStreamSynchronize(s->stream));  // the old graph may still run
        build_step_graph<R, NF>(g, a, EQ_GIVEN, s->lanes, s->d_flags);
        f = {a.x, a.rhs, a.As_od};
    }
    FEA_CUDA_TRY(cudaGraphLaunch(g.exec, s->stream));
}

// u0, t: solver-order device arrays.  Leaves lam = dJ/du0 (solver order) and
// gD = dJ/dD (FP64, per element) when `grads`, and the handle's field at u_N.
template <typename R>
double adjoint_core(fea_solver* s, const R* u0, const R* t, int64_t nsteps, int64_t ckpt, bool grads, R* lam,
                    double* gD) {
    if (step_kind(s->prm) != EQ_ADV_EXPLICIT) {
        set_error("the adjoint needs equation FEA_ADVECTION_DIFFUSION with advection_scheme 1");
        throw Error{FEA_ERR_STATE};
    }
    cudaStream_t st = s->stream;
    const CallRuns runs(s);
    const int64_t N = s->N;
    const size_t rb = sizeof(R) * (size_t)N;
    const auto d2d = cudaMemcpyDeviceToDevice;
    ckpt = std::min(ckpt, nsteps);
    const int64_t nck = ceil_div(nsteps, ckpt);
    ensure_layout<R>(s, false);
    const SweepStates states(s->scratch[3]);
    Scratch& tmp = s->scratch[0];
    tmp.rewind();
    R* ck = states.mem.alloc<R>(nck * N);
    R* seg = states.mem.alloc<R>((ckpt + 1) * N);
    R* mu = tmp.alloc<R>(pad_tiles(N));  // x of the solves: whole tiles
    R* uN = tmp.alloc<R>(N);
    R* lam_f = lam ? lam : tmp.alloc<R>(N);
    double* J = tmp.alloc<double>(1);
    R* u = (R*)s->F.u;
    FEA_CUDA_TRY(cudaMemcpyAsync(u, u0, rb, d2d, st));
    for (int64_t sg = 0; sg < nck; sg++) {  // forward sweep, a checkpoint per segment
        FEA_CUDA_TRY(cudaMemcpyAsync(ck + sg * N, u, rb, d2d, st));
        advance<R>(s, std::min(ckpt, nsteps - sg * ckpt));
    }
    FEA_CUDA_TRY(cudaMemcpyAsync(uN, u, rb, d2d, st));
    adjoint_loss<R>(s->Pc, (const R*)s->Mc, u, t, lam_f, s->d_part, max_grid_blocks(), s->d_tickets + 5, J, st);
    if (grads) {
        FEA_CUDA_TRY(cudaMemsetAsync(gD, 0, sizeof(double) * (size_t)s->T, st));
        FEA_CUDA_TRY(cudaMemsetAsync(mu, 0, sizeof(R) * (size_t)pad_tiles(N), st));
        StepArgs<R, 1> a = make_args<R, 1>(s, false);
        a.x = (FV<R, 1>*)mu;
        a.rhs = (const FV<R, 1>*)lam_f;
        const double dt = time_step(s->prm), c = s->prm.advdiff_c, sign = s->prm.advection_sign;
        try {
            for (int64_t sg = nck - 1; sg >= 0; sg--) {
                const int64_t n0 = sg * ckpt, n1 = std::min(n0 + ckpt, nsteps);
                FEA_CUDA_TRY(cudaMemcpyAsync(u, ck + sg * N, rb, d2d, st));
                for (int64_t n = n0; n < n1; n++) {  // u^{n0+1} .. u^{n1}
                    advance<R>(s, 1);
                    FEA_CUDA_TRY(cudaMemcpyAsync(seg + (n - n0 + 1) * N, u, rb, d2d, st));
                }
                for (int64_t n = n1 - 1; n >= n0; n--) {
                    run_given<R, 1>(s, a);  // mu = A^-1 lam, warm-started from the previous mu
                    adjoint_grad_D<R>(s->Kloc, s->tri, s->idx_c, s->T, c, mu, seg + (n - n0 + 1) * N, gD, st);
                    adjoint_lambda<R>(s->Pc, (const R*)s->Mc, (const R*)s->Advc, dt, sign, mu, lam_f, st);
                }
            }
        } catch (...) {
            cudaStreamSynchronize(st);
            throw;
        }
    }
    FEA_CUDA_TRY(cudaMemcpyAsync(u, uN, rb, d2d, st));
    return sweep_result(s, J);
}

// ---- adjoint of the mass-weighted Gray-Scott step (kernels in adjoint.cu) ---------
// x0, t: solver-order (u, v) pairs; use_u / use_v select the loss terms.
// Leaves lam = (dJ/du0, dJ/dv0) in solver order, adds (dJ/dF, dJ/dk, dJ/dDu,
// dJ/dDv) into g[4] (device), and the handle's fields at the final state.
template <typename R>
double adjoint_gs_core(fea_solver* s, const FV<R, 2>* x0, const FV<R, 2>* t, int use_u, int use_v, int64_t nsteps,
                       int64_t ckpt, bool grads, FV<R, 2>* lam, double* g) {
    if (step_kind(s->prm) != EQ_GS_CONSISTENT) {
        set_error("the Gray-Scott adjoint needs equation FEA_REACTION_DIFFUSION with reaction_mode 1");
        throw Error{FEA_ERR_STATE};
    }
    const GuessOff guess_off(s);  // recomputed forward states must equal the forward sweep's
    const DiagonalOnly diagonal(s, sizeof(R) == 4);
    cudaStream_t st = s->stream;
    const CallRuns runs(s);
    const int64_t N = s->N;
    const size_t xb = sizeof(FV<R, 2>) * (size_t)N;
    const auto d2d = cudaMemcpyDeviceToDevice;
    ckpt = std::min(ckpt, nsteps);
    const int64_t nck = ceil_div(nsteps, ckpt);
    ensure_layout<R>(s, true);  // the forward steps update the operator to the current parameters
    const SweepStates states(s->scratch[3]);
    Scratch& tmp = s->scratch[0];
    tmp.rewind();
    FV<R, 2>* ck = states.mem.alloc<FV<R, 2>>(nck * N);
    FV<R, 2>* seg = states.mem.alloc<FV<R, 2>>((ckpt + 1) * N);
    FV<R, 2>* mu = tmp.alloc<FV<R, 2>>(pad_tiles(N));  // x of the solves: whole tiles
    FV<R, 2>* xN = tmp.alloc<FV<R, 2>>(N);
    double* J = tmp.alloc<double>(1);
    FV<R, 2>* x = (FV<R, 2>*)s->F.uv;
    FEA_CUDA_TRY(cudaMemcpyAsync(x, x0, xb, d2d, st));
    for (int64_t sg = 0; sg < nck; sg++) {  // forward sweep, a checkpoint per segment
        FEA_CUDA_TRY(cudaMemcpyAsync(ck + sg * N, x, xb, d2d, st));
        advance<R>(s, std::min(ckpt, nsteps - sg * ckpt));
    }
    FEA_CUDA_TRY(cudaMemcpyAsync(xN, x, xb, d2d, st));
    adjoint_gs_loss<R>(s->Pc, (const R*)s->Mc, x, t, use_u, use_v, lam, s->d_part, max_grid_blocks(),
                       s->d_tickets + 5, J, st);
    if (grads) {
        FEA_CUDA_TRY(cudaMemsetAsync(mu, 0, sizeof(FV<R, 2>) * (size_t)pad_tiles(N), st));
        StepArgs<R, 2> a = make_args<R, 2>(s, false);
        a.x = mu;
        a.rhs = lam;
        const fea_params& p = s->prm;
        const double dt = p.rd_time_step, F = p.rd_feed_rate, kr = p.rd_kill_rate;
        try {
            for (int64_t sg = nck - 1; sg >= 0; sg--) {
                const int64_t n0 = sg * ckpt, n1 = std::min(n0 + ckpt, nsteps);
                FEA_CUDA_TRY(cudaMemcpyAsync(x, ck + sg * N, xb, d2d, st));
                FEA_CUDA_TRY(cudaMemcpyAsync(seg, x, xb, d2d, st));
                for (int64_t n = n0; n < n1; n++) {  // x^{n0+1} .. x^{n1}
                    advance<R>(s, 1);
                    FEA_CUDA_TRY(cudaMemcpyAsync(seg + (n - n0 + 1) * N, x, xb, d2d, st));
                }
                for (int64_t n = n1 - 1; n >= n0; n--) {
                    run_given<R, 2>(s, a);  // mu = A^-1 lam (both fields), warm-started
                    adjoint_gs_step<R>(s->Pc, (const R*)s->Mc, (const R*)s->Kc, mu, seg + (n - n0) * N,
                                       seg + (n - n0 + 1) * N, dt, F, kr, lam, s->d_part, max_grid_blocks(),
                                       s->d_tickets + 6, g, st);
                }
            }
        } catch (...) {
            cudaStreamSynchronize(st);
            throw;
        }
    }
    FEA_CUDA_TRY(cudaMemcpyAsync(x, xN, xb, d2d, st));
    return sweep_result(s, J);
}

// Node-indexed float arrays (NULL targets drop their loss terms).
template <typename R>
void adjoint_gs_host(fea_solver* s, const float* u0, const float* v0, const float* tu, const float* tv,
                     int64_t nsteps, int64_t ckpt, double* loss, float* gu, float* gv, double* gparams) {
    cudaStream_t st = s->stream;
    const int64_t N = s->N, V = s->V;
    Scratch& tmp = s->scratch[1];
    tmp.rewind();
    FV<R, 2>* x0 = tmp.alloc<FV<R, 2>>(N);
    FV<R, 2>* t = tmp.alloc<FV<R, 2>>(N);
    FV<R, 2>* lam = tmp.alloc<FV<R, 2>>(N);
    double* g = tmp.alloc<double>(4);
    FEA_CUDA_TRY(cudaMemsetAsync(t, 0, sizeof(FV<R, 2>) * (size_t)N, st));
    FEA_CUDA_TRY(cudaMemsetAsync(g, 0, 4 * sizeof(double), st));
    const std::pair<const float*, std::pair<R*, int>> ins[4] = {
        {u0, {(R*)x0, 0}}, {v0, {(R*)x0, 1}}, {tu, {(R*)t, 0}}, {tv, {(R*)t, 1}}};
    for (const auto& in : ins) {
        if (!in.first) continue;
        FEA_CUDA_TRY(cudaMemcpyAsync(s->d_nodes, in.first, sizeof(float) * V, cudaMemcpyHostToDevice, st));
        k_gather_nodes<R><<<launch_grid(V), kBlock, 0, st>>>(s->d_nodes, s->idx_c, V, in.second.first, 2,
                                                              in.second.second, nullptr);
        FEA_CHECK_LAUNCH();
    }
    const bool grads = gu || gv || gparams;
    const double J = adjoint_gs_core<R>(s, x0, t, tu != nullptr, tv != nullptr, nsteps, ckpt, grads, lam, g);
    if (loss) *loss = J;
    float* outs[2] = {gu, gv};
    for (int f = 0; f < 2; f++) {
        if (!outs[f]) continue;
        k_scatter_nodes<R><<<launch_grid(V), kBlock, 0, st>>>((const R*)lam, s->idx_c, V, s->d_nodes, 2, f);
        FEA_CHECK_LAUNCH();
        FEA_CUDA_TRY(cudaMemcpyAsync(outs[f], s->d_nodes, sizeof(float) * V, cudaMemcpyDeviceToHost, st));
        FEA_CUDA_TRY(cudaStreamSynchronize(st));
    }
    if (gparams) FEA_CUDA_TRY(cudaMemcpyAsync(gparams, g, 4 * sizeof(double), cudaMemcpyDeviceToHost, st));
    FEA_CUDA_TRY(cudaStreamSynchronize(st));
}

// Unknown-indexed device arrays in the handle's precision.
template <typename R>
void adjoint_gs_device(fea_solver* s, const void* u0, const void* v0, const void* tu, const void* tv,
                       int64_t nsteps, int64_t ckpt, double* loss, void* gu, void* gv, double* gparams) {
    cudaStream_t st = s->stream;
    const int64_t N = s->N;
    Scratch& tmp = s->scratch[1];
    tmp.rewind();
    FV<R, 2>* x0 = tmp.alloc<FV<R, 2>>(N);
    FV<R, 2>* t = tmp.alloc<FV<R, 2>>(N);
    FV<R, 2>* lam = tmp.alloc<FV<R, 2>>(N);
    double* g = tmp.alloc<double>(4);
    FEA_CUDA_TRY(cudaMemsetAsync(t, 0, sizeof(FV<R, 2>) * (size_t)N, st));
    FEA_CUDA_TRY(cudaMemsetAsync(g, 0, 4 * sizeof(double), st));
    const std::pair<const void*, std::pair<R*, int>> ins[4] = {
        {u0, {(R*)x0, 0}}, {v0, {(R*)x0, 1}}, {tu, {(R*)t, 0}}, {tv, {(R*)t, 1}}};
    if (N > 0)
        for (const auto& in : ins) {
            if (!in.first) continue;
            k_copy_to_state<R><<<launch_grid(N), kBlock, 0, st>>>((const R*)in.first, s->pos, N, in.second.first, 2,
                                                                   in.second.second, nullptr);
            FEA_CHECK_LAUNCH();
        }
    const bool grads = gu || gv || gparams;
    const double J = adjoint_gs_core<R>(s, x0, t, tu != nullptr, tv != nullptr, nsteps, ckpt, grads, lam, g);
    if (loss) *loss = J;
    void* outs[2] = {gu, gv};
    for (int f = 0; f < 2; f++)
        if (outs[f] && N > 0) {
            k_copy_from_state<R><<<launch_grid(N), kBlock, 0, st>>>((const R*)lam, s->pos, N, (R*)outs[f], 2, f);
            FEA_CHECK_LAUNCH();
        }
    if (gparams) FEA_CUDA_TRY(cudaMemcpyAsync(gparams, g, 4 * sizeof(double), cudaMemcpyDeviceToHost, st));
    FEA_CUDA_TRY(cudaStreamSynchronize(st));
}

// Node-indexed float inputs and outputs (the host entry point).
template <typename R>
void adjoint_host(fea_solver* s, const float* u0, const float* target, int64_t nsteps, int64_t ckpt, double* loss,
                  float* grad_u0, float* grad_D) {
    cudaStream_t st = s->stream;
    const int64_t N = s->N, V = s->V, T = s->T;
    Scratch& tmp = s->scratch[1];
    tmp.rewind();
    R* u0s = tmp.alloc<R>(N);
    R* ts = tmp.alloc<R>(N);
    R* lam = tmp.alloc<R>(N);
    double* gD = tmp.alloc<double>(T);
    float* gDf = tmp.alloc<float>(T);
    const std::pair<const float*, R*> ins[2] = {{u0, u0s}, {target, ts}};
    for (const auto& in : ins) {
        FEA_CUDA_TRY(cudaMemcpyAsync(s->d_nodes, in.first, sizeof(float) * V, cudaMemcpyHostToDevice, st));
        k_gather_nodes<R><<<launch_grid(V), kBlock, 0, st>>>(s->d_nodes, s->idx_c, V, in.second, 1, 0, nullptr);
        FEA_CHECK_LAUNCH();
    }
    const bool grads = grad_u0 || grad_D;
    const double J = adjoint_core<R>(s, u0s, ts, nsteps, ckpt, grads, lam, gD);
    if (loss) *loss = J;
    if (grad_u0) {
        k_scatter_nodes<R><<<launch_grid(V), kBlock, 0, st>>>(lam, s->idx_c, V, s->d_nodes, 1, 0);
        FEA_CHECK_LAUNCH();
        FEA_CUDA_TRY(cudaMemcpyAsync(grad_u0, s->d_nodes, sizeof(float) * V, cudaMemcpyDeviceToHost, st));
    }
    if (grad_D) {
        k_convert<double, float><<<launch_grid(T), kBlock, 0, st>>>(gD, T, gDf);
        FEA_CHECK_LAUNCH();
        FEA_CUDA_TRY(cudaMemcpyAsync(grad_D, gDf, sizeof(float) * T, cudaMemcpyDeviceToHost, st));
    }
    FEA_CUDA_TRY(cudaStreamSynchronize(st));
}

// Unknown-indexed device arrays in the handle's precision.
template <typename R>
void adjoint_device(fea_solver* s, const void* u0, const void* target, int64_t nsteps, int64_t ckpt, double* loss,
                    void* grad_u0, void* grad_D) {
    cudaStream_t st = s->stream;
    const int64_t N = s->N, T = s->T;
    Scratch& tmp = s->scratch[1];
    tmp.rewind();
    R* u0s = tmp.alloc<R>(N);
    R* ts = tmp.alloc<R>(N);
    R* lam = tmp.alloc<R>(N);
    double* gD = tmp.alloc<double>(T);
    if (N > 0) {
        k_copy_to_state<R><<<launch_grid(N), kBlock, 0, st>>>((const R*)u0, s->pos, N, u0s, 1, 0, nullptr);
        k_copy_to_state<R><<<launch_grid(N), kBlock, 0, st>>>((const R*)target, s->pos, N, ts, 1, 0, nullptr);
        FEA_CHECK_LAUNCH();
    }
    const bool grads = grad_u0 || grad_D;
    const double J = adjoint_core<R>(s, u0s, ts, nsteps, ckpt, grads, lam, gD);
    if (loss) *loss = J;
    if (grad_u0 && N > 0) {
        k_copy_from_state<R><<<launch_grid(N), kBlock, 0, st>>>(lam, s->pos, N, (R*)grad_u0, 1, 0);
        FEA_CHECK_LAUNCH();
    }
    if (grad_D) {
        k_convert<double, R><<<launch_grid(T), kBlock, 0, st>>>(gD, T, (R*)grad_D);
        FEA_CHECK_LAUNCH();
    }
    FEA_CUDA_TRY(cudaStreamSynchronize(st));
}

}  // namespace

MeshView mesh_view(const fea_solver* s) {
    MeshView m;
    m.V = s->V;
    m.T = s->T;
    m.N = s->N;
    m.Pc = &s->Pc;
    m.emap = s->emap;
    m.M64 = s->M64;
    m.K64 = s->K64;
    m.Adv64 = s->Adv64;
    m.idx_c = s->idx_c;
    m.stream = s->stream;
    return m;
}

// ---- after the solve: smooth normals and the .ply export ----------------------------

// The displayed field (v for Gray-Scott, u otherwise; 0 on Dirichlet points),
// node-indexed, into the handle's staging buffer.
void stage_node_values(fea_solver* s) {
    const int which = displayed_field(s->prm);
    Fields& F = s->F;
    const int64_t V = s->V;
    if (s->precision == FEA_FP64) {
        if (F.interleaved)
            k_scatter_nodes<double><<<launch_grid(V), kBlock, 0, s->stream>>>((double*)F.uv, s->idx_c, V, s->d_nodes,
                                                                               2, which);
        else
            k_scatter_nodes<double><<<launch_grid(V), kBlock, 0, s->stream>>>(
                (double*)(which ? F.v : F.u), s->idx_c, V, s->d_nodes, 1, 0);
    } else {
        if (F.interleaved)
            k_scatter_nodes<float><<<launch_grid(V), kBlock, 0, s->stream>>>((float*)F.uv, s->idx_c, V, s->d_nodes, 2,
                                                                              which);
        else
            k_scatter_nodes<float><<<launch_grid(V), kBlock, 0, s->stream>>>((float*)(which ? F.v : F.u), s->idx_c,
                                                                              V, s->d_nodes, 1, 0);
    }
    FEA_CHECK_LAUNCH();
}

void ensure_vertex_triangles(fea_solver* s) {
    if (s->vt_ptr) return;
    s->vt_ptr = s->mesh_mem.alloc<int32_t>(s->V + 1);
    s->vt_tri = s->mesh_mem.alloc<int32_t>(3 * s->T);
    build_vertex_triangles(s->tri, s->T, s->V, s->vt_ptr, s->vt_tri, s->stream);
}

// nrm and out: device float[3V]; face: float[3T] scratch
void smooth_normals_dev(fea_solver* s, const float* nrm, float e, float* face, float* out) {
    ensure_vertex_triangles(s);
    stage_node_values(s);
    smooth_normals(s->xyz, s->tri, s->T, s->V, s->vt_ptr, s->vt_tri, nrm, s->d_nodes, e, face, out, s->stream);
}

struct PlyGeometry {
    std::vector<float> pos, val;
    std::vector<uint32_t> tri;
};

struct PosKey {
    uint32_t b[3];
    bool operator==(const PosKey& o) const { return b[0] == o.b[0] && b[1] == o.b[1] && b[2] == o.b[2]; }
};
struct PosKeyHash {
    size_t operator()(const PosKey& k) const {
        uint64_t h = 1469598103934665603ull;
        for (uint32_t x : k.b) h = (h ^ x) * 1099511628211ull;
        return (size_t)h;
    }
};

uint32_t key_bits(float f) {
    if (f == 0.0f) f = 0.0f;  // -0 and +0 are the same position
    uint32_t u;
    memcpy(&u, &f, 4);
    return u;
}

// Clipping on the device, then the reference's first-seen numbering of the
// positions (an exact-equality position map) on the host.
void ply_geometry(fea_solver* s, const float* nrm_host, float e, float thr, int mesh_type, PlyGeometry& g) {
    const int64_t V = s->V, T = s->T;
    cudaStream_t st = s->stream;
    DeviceArena tmp;
    float* nrm = tmp.alloc<float>(3 * V);
    float* pos = tmp.alloc<float>(18 * T);
    float* pval = tmp.alloc<float>(6 * T);
    uint8_t* used = tmp.alloc<uint8_t>(6 * T);
    int32_t* otri = tmp.alloc<int32_t>(12 * T);
    FEA_CUDA_TRY(cudaMemcpyAsync(nrm, nrm_host, sizeof(float) * 3 * V, cudaMemcpyHostToDevice, st));
    stage_node_values(s);
    ply_clip(s->xyz, s->tri, T, nrm, s->d_nodes, e, thr, mesh_type, pos, pval, used, otri, st);
    std::vector<float> hpos(18 * T), hval(6 * T);
    std::vector<uint8_t> hused(6 * T);
    std::vector<int32_t> htri(12 * T);
    FEA_CUDA_TRY(cudaMemcpyAsync(hpos.data(), pos, sizeof(float) * 18 * T, cudaMemcpyDeviceToHost, st));
    FEA_CUDA_TRY(cudaMemcpyAsync(hval.data(), pval, sizeof(float) * 6 * T, cudaMemcpyDeviceToHost, st));
    FEA_CUDA_TRY(cudaMemcpyAsync(hused.data(), used, 6 * T, cudaMemcpyDeviceToHost, st));
    FEA_CUDA_TRY(cudaMemcpyAsync(htri.data(), otri, sizeof(int32_t) * 12 * T, cudaMemcpyDeviceToHost, st));
    FEA_CUDA_TRY(cudaStreamSynchronize(st));
    std::unordered_map<PosKey, uint32_t, PosKeyHash> map;
    std::vector<uint32_t> slot_idx(6 * T, 0);
    g.pos.clear();
    g.val.clear();
    g.tri.clear();
    for (int64_t k = 0; k < T; k++) {
        for (int j = 0; j < 6; j++) {  // the order of the reference's add_clipped_position calls
            const int64_t q = 6 * k + j;
            if (!hused[q]) continue;
            const float* p = &hpos[3 * q];
            const PosKey key{{key_bits(p[0]), key_bits(p[1]), key_bits(p[2])}};
            auto it = map.find(key);
            if (it == map.end()) {
                const uint32_t idx = (uint32_t)g.val.size();
                map.emplace(key, idx);
                g.pos.insert(g.pos.end(), p, p + 3);
                g.val.push_back(hval[q]);
                slot_idx[q] = idx;
            } else {
                slot_idx[q] = it->second;
            }
        }
        for (int m = 0; m < 4; m++) {
            const int32_t* t3 = &htri[12 * k + 3 * m];
            if (t3[0] < 0) continue;
            for (int i = 0; i < 3; i++) g.tri.push_back(slot_idx[t3[i]]);
        }
    }
}

void append_float(std::string& out, float x) {
    char buf[64];
    const auto r = std::to_chars(buf, buf + sizeof(buf), x);  // shortest round-trip form, as std::format("{}")
    out.append(buf, r.ptr);
}

// Surface::export_to_ply's file (Surface.cpp:254-284): ASCII PLY, float
// x y z red green blue per vertex (color from the polynomial color map,
// ColorMap::get_color, ColorMap.cpp:12-14), "3 a b c" per face.
void write_ply(const char* path, const PlyGeometry& g, const float* coeffs) {
    std::string out;
    const size_t nv = g.val.size(), nf = g.tri.size() / 3;
    out.reserve(64 * nv + 24 * nf + 256);
    out += "ply\nformat ascii 1.0\nelement vertex " + std::to_string(nv) +
           "\nproperty float x\nproperty float y\nproperty float z\nproperty float red\nproperty float green\n"
           "property float blue\nelement face " +
           std::to_string(nf) + "\nproperty list uchar uint vertex_indices\nend_header\n";
    for (size_t i = 0; i < nv; i++) {
        const float t = g.val[i];
        float col[3];
        for (int ch = 0; ch < 3; ch++) {  // c0 + t (c1 + t (c2 + ... + t c6))
            float acc = coeffs[3 * 6 + ch];
            for (int k = 5; k >= 0; k--) acc = coeffs[3 * k + ch] + t * acc;
            col[ch] = acc;
        }
        const float v6[6] = {g.pos[3 * i], g.pos[3 * i + 1], g.pos[3 * i + 2], col[0], col[1], col[2]};
        for (int j = 0; j < 6; j++) {
            append_float(out, v6[j]);
            out += j < 5 ? ' ' : '\n';
        }
    }
    for (size_t f = 0; f < nf; f++)
        out += "3 " + std::to_string(g.tri[3 * f]) + " " + std::to_string(g.tri[3 * f + 1]) + " " +
               std::to_string(g.tri[3 * f + 2]) + "\n";
    FILE* fh = fopen(path, "wb");
    if (!fh) {
        set_error("cannot open %s for writing", path);
        throw Error{FEA_ERR_INVALID_ARGUMENT};
    }
    const size_t wrote = fwrite(out.data(), 1, out.size(), fh);
    const int closed = fclose(fh);
    if (wrote != out.size() || closed != 0) {
        set_error("writing %s failed", path);
        throw Error{FEA_ERR_INVALID_ARGUMENT};
    }
}

// Device partial-reduction storage sized for the widest grid.
void alloc_run_state(fea_solver* s) {
    s->d_prm = s->run_mem.alloc<StepParams>(1);
    s->d_cg = s->run_mem.alloc<CgState>(2);
    s->d_run = s->run_mem.alloc<RunState>(1);
    s->d_part = s->run_mem.alloc<double>(16 * (int64_t)max_grid_blocks());
    s->d_tickets = s->run_mem.alloc<unsigned int>(8);
    s->d_flags = s->run_mem.alloc<LoopFlags>(1);
    FEA_CUDA_TRY(cudaMemsetAsync(s->d_flags, 0, sizeof(LoopFlags), s->stream));
    const char* mode = getenv("FEA_LAUNCH_MODE");
    s->stream_mode = mode && strcmp(mode, "stream") == 0;
    FEA_CUDA_TRY(cudaMemsetAsync(s->d_cg, 0, 2 * sizeof(CgState), s->stream));
    FEA_CUDA_TRY(cudaMemsetAsync(s->d_run, 0, sizeof(RunState), s->stream));
    FEA_CUDA_TRY(cudaMemsetAsync(s->d_tickets, 0, 8 * sizeof(unsigned int), s->stream));
    FEA_CUDA_TRY(cudaMallocHost(&s->h_run, sizeof(RunState)));
}

}  // namespace fea

#define API_BEGIN try {
#define API_END                                                          \
    }                                                                    \
    catch (const fea::Error& e) {                                        \
        return e.code;                                                   \
    }                                                                    \
    catch (const std::bad_alloc&) {                                      \
        return fea::fail(FEA_ERR_OUT_OF_MEMORY, "host allocation failed"); \
    }                                                                    \
    catch (...) {                                                        \
        return fea::fail(FEA_ERR_CUDA, "unexpected failure");            \
    }                                                                    \
    return FEA_OK;

extern "C" {

const char* fea_last_error(void) { return fea::g_err; }
const char* fea_version(void) { return "fea_gb300 1.0 (sm_103a)"; }

int fea_params_default(fea_params* o) {
    if (!o) return fail(FEA_ERR_INVALID_ARGUMENT, "null params");
    memset(o, 0, sizeof(*o));
    o->equation = FEA_WAVE;  // FEMContext.hpp:31
    o->heat_time_step = 0.01f;
    o->heat_conductivity = 0.05f;
    o->advdiff_time_step = 0.001f;
    o->advdiff_c = 0.25f;
    o->advdiff_velocity[0] = 1.0f;
    o->wave_time_step = 0.05f;
    o->wave_c = 0.05f;
    o->rd_time_step = 0.001f;
    o->rd_Du = 0.08f;
    o->rd_Dv = 0.04f;
    o->rd_feed_rate = 0.035f;
    o->rd_kill_rate = 0.06f;
    o->reaction_mode = 0;
    o->wave_scheme = 0;
    o->newmark_beta = 0.25;
    o->newmark_gamma = 0.5;
    o->advection_scheme = 0;
    o->advection_sign = 1.0f;
    o->velocity_mode = 0;
    o->cg_tolerance = 0.0;
    o->cg_max_iterations = 0;
    o->cg_refine = 1;
    o->cg_initial_guess = 0;
    return FEA_OK;
}

int fea_create(const float* vertices, int64_t V, const uint32_t* triangles, int64_t T, const uint8_t* on_boundary,
               int bc, int precision, const fea_params* params, fea_solver** out) {
    if (!out) return fail(FEA_ERR_INVALID_ARGUMENT, "null output handle");
    *out = nullptr;
    if (!vertices || !triangles || V <= 0 || T <= 0)
        return fail(FEA_ERR_BAD_MESH, "mesh must have vertices and triangles");
    if (bc != FEA_DIRICHLET && bc != FEA_NEUMANN) return fail(FEA_ERR_INVALID_ARGUMENT, "bad boundary condition");
    if (precision != FEA_FP32 && precision != FEA_FP64) return fail(FEA_ERR_INVALID_ARGUMENT, "bad precision");
    if (V >= (int64_t)INT32_MAX || 9 * T >= (int64_t)INT32_MAX) return fail(FEA_ERR_TOO_LARGE, "mesh exceeds int32 indexing");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return fail(FEA_ERR_NO_DEVICE, "no CUDA device");
    fea_solver* s = nullptr;
    API_BEGIN
    s = new fea_solver();
    FEA_CUDA_TRY(cudaGetDevice(&s->device));
    FEA_CUDA_TRY(cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking));
    s->precision = precision;
    s->bc = bc;
    s->V = V;
    s->T = T;
    if (params) s->prm = *params;
    else fea_params_default(&s->prm);
    s->xyz = s->mesh_mem.alloc<float>(3 * V);
    s->tri = s->mesh_mem.alloc<uint32_t>(3 * T);
    s->ob = s->mesh_mem.alloc<uint8_t>(V);
    s->d_nodes = s->mesh_mem.alloc<float>(V);
    FEA_CUDA_TRY(cudaMemcpyAsync(s->xyz, vertices, sizeof(float) * 3 * V, cudaMemcpyHostToDevice, s->stream));
    FEA_CUDA_TRY(cudaMemcpyAsync(s->tri, triangles, sizeof(uint32_t) * 3 * T, cudaMemcpyHostToDevice, s->stream));
    if (const int bad = check_mesh(s->xyz, s->tri, T, V, s->stream)) {
        fea_destroy(s);
        return fail(FEA_ERR_BAD_MESH, (bad & 1)   ? "triangle index out of range"
                                      : (bad & 2) ? "non-finite vertex coordinate"
                                                  : "degenerate triangle (zero area)");
    }
    if (on_boundary) {
        FEA_CUDA_TRY(cudaMemcpyAsync(s->ob, on_boundary, V, cudaMemcpyHostToDevice, s->stream));
    } else {
        detect_boundary(s->tri, T, V, s->ob, s->stream);
    }
    {
        std::vector<uint8_t> h(V);
        FEA_CUDA_TRY(cudaMemcpyAsync(h.data(), s->ob, V, cudaMemcpyDeviceToHost, s->stream));
        FEA_CUDA_TRY(cudaStreamSynchronize(s->stream));
        int64_t nb = 0;
        for (int64_t i = 0; i < V; i++) nb += h[i] ? 1 : 0;
        s->nb = nb;
    }
    alloc_run_state(s);
    build_context(s);
    if (precision == FEA_FP64) upload_params<double>(s);
    else upload_params<float>(s);
    *out = s;
    return FEA_OK;
    }
    catch (const fea::Error& e) {
        if (s) fea_destroy(s);
        return e.code;
    }
    catch (const std::bad_alloc&) {
        if (s) fea_destroy(s);
        return fail(FEA_ERR_OUT_OF_MEMORY, "host allocation failed");
    }
    catch (...) {
        if (s) fea_destroy(s);
        return fail(FEA_ERR_CUDA, "unexpected failure");
    }
}

int fea_destroy(fea_solver* s) {
    if (!s) return FEA_OK;
    cudaSetDevice(s->device);
    if (s->stream) cudaStreamSynchronize(s->stream);
    s->graph.destroy();
    s->init_graph.destroy();
    s->diag_graph.destroy();
    for (auto& g : s->given_graph) g.destroy();
    s->mat_mem.release();
    s->run_mem.release();
    s->mesh_mem.release();
    for (Scratch& k : s->scratch) k.release();
    if (s->h_run) cudaFreeHost(s->h_run);
    if (s->stream) cudaStreamDestroy(s->stream);
    delete s;
    return FEA_OK;
}

int fea_set_boundary_condition(fea_solver* s, int bc) {
    API_BEGIN
    check_handle(s);
    if (bc != FEA_DIRICHLET && bc != FEA_NEUMANN) return fail(FEA_ERR_INVALID_ARGUMENT, "bad boundary condition");
    FEA_CUDA_TRY(cudaStreamSynchronize(s->stream));
    s->bc = bc;
    build_context(s);
    s->op_dirty = true;
    if (s->precision == FEA_FP64) upload_params<double>(s);
    else upload_params<float>(s);
    API_END
}

int fea_set_params(fea_solver* s, const fea_params* p) {
    API_BEGIN
    check_handle(s);
    if (!p) return fail(FEA_ERR_INVALID_ARGUMENT, "null params");
    if (p->equation < FEA_HEAT || p->equation > FEA_REACTION_DIFFUSION)
        return fail(FEA_ERR_INVALID_ARGUMENT, "bad equation");
    FEA_CUDA_TRY(cudaStreamSynchronize(s->stream));
    const bool wave_changed = p->wave_c != s->prm.wave_c || p->wave_time_step != s->prm.wave_time_step ||
                              p->newmark_beta != s->prm.newmark_beta;
    if (wave_changed) s->acc_valid = false;
    s->prm = *p;
    s->op_dirty = true;
    if (s->precision == FEA_FP64) upload_params<double>(s);
    else upload_params<float>(s);
    API_END
}

int fea_set_element_fields(fea_solver* s, const float* diffusivity, const float* velocity) {
    API_BEGIN
    check_handle(s);
    FEA_CUDA_TRY(cudaStreamSynchronize(s->stream));
    if (diffusivity) {
        if (!s->elem_D) {
            s->elem_D = s->mesh_mem.alloc<float>(s->T);
            s->elem_Dr = s->mesh_mem.alloc<double>(s->T);
        }
        FEA_CUDA_TRY(cudaMemcpyAsync(s->elem_D, diffusivity, sizeof(float) * s->T, cudaMemcpyHostToDevice, s->stream));
        k_float_to<double><<<launch_grid(s->T), kBlock, 0, s->stream>>>(s->elem_D, s->T, s->elem_Dr);
        FEA_CHECK_LAUNCH();
    }
    if (velocity) {
        if (!s->elem_vel) s->elem_vel = s->mesh_mem.alloc<float>(3 * s->T);
        FEA_CUDA_TRY(cudaMemcpyAsync(s->elem_vel, velocity, sizeof(float) * 3 * s->T, cudaMemcpyHostToDevice,
                                     s->stream));
    }
    assemble(s);
    FEA_CUDA_TRY(cudaStreamSynchronize(s->stream));
    API_END
}

int fea_set_element_diffusivity_device(fea_solver* s, const void* diffusivity) {
    API_BEGIN
    check_handle(s);
    if (!diffusivity) return fail(FEA_ERR_INVALID_ARGUMENT, "null diffusivity");
    FEA_CUDA_TRY(cudaStreamSynchronize(s->stream));
    if (!s->elem_D) {
        s->elem_D = s->mesh_mem.alloc<float>(s->T);
        s->elem_Dr = s->mesh_mem.alloc<double>(s->T);
    }
    if (s->precision == FEA_FP64) {
        FEA_CUDA_TRY(cudaMemcpyAsync(s->elem_Dr, diffusivity, sizeof(double) * s->T, cudaMemcpyDeviceToDevice,
                                     s->stream));
        k_convert<double, float><<<launch_grid(s->T), kBlock, 0, s->stream>>>(s->elem_Dr, s->T, s->elem_D);
    } else {
        FEA_CUDA_TRY(cudaMemcpyAsync(s->elem_D, diffusivity, sizeof(float) * s->T, cudaMemcpyDeviceToDevice,
                                     s->stream));
        k_float_to<double><<<launch_grid(s->T), kBlock, 0, s->stream>>>(s->elem_D, s->T, s->elem_Dr);
    }
    FEA_CHECK_LAUNCH();
    assemble(s);
    FEA_CUDA_TRY(cudaStreamSynchronize(s->stream));
    API_END
}

int fea_adjoint_advdiff(fea_solver* s, const float* u0, const float* target, int64_t nsteps,
                        int64_t checkpoint_every, double* loss, float* grad_u0, float* grad_D) {
    API_BEGIN
    check_handle(s);
    if (!u0 || !target || nsteps < 1 || checkpoint_every < 1)
        return fail(FEA_ERR_INVALID_ARGUMENT, "adjoint needs u0, target, nsteps >= 1 and checkpoint_every >= 1");
    if (s->precision == FEA_FP64) adjoint_host<double>(s, u0, target, nsteps, checkpoint_every, loss, grad_u0, grad_D);
    else adjoint_host<float>(s, u0, target, nsteps, checkpoint_every, loss, grad_u0, grad_D);
    API_END
}

int fea_adjoint_advdiff_device(fea_solver* s, const void* u0, const void* target, int64_t nsteps,
                               int64_t checkpoint_every, double* loss, void* grad_u0, void* grad_D) {
    API_BEGIN
    check_handle(s);
    if (!u0 || !target || nsteps < 1 || checkpoint_every < 1)
        return fail(FEA_ERR_INVALID_ARGUMENT, "adjoint needs u0, target, nsteps >= 1 and checkpoint_every >= 1");
    if (s->precision == FEA_FP64)
        adjoint_device<double>(s, u0, target, nsteps, checkpoint_every, loss, grad_u0, grad_D);
    else adjoint_device<float>(s, u0, target, nsteps, checkpoint_every, loss, grad_u0, grad_D);
    API_END
}

int fea_smooth_normals(fea_solver* s, const float* normals, float vertex_extrusion, float* out) {
    API_BEGIN
    check_handle(s);
    if (!normals || !out) return fail(FEA_ERR_INVALID_ARGUMENT, "null normals or output");
    Scratch& tmp = s->scratch[2];
    tmp.rewind();
    float* face = tmp.alloc<float>(3 * s->T);
    float* nrm = tmp.alloc<float>(3 * s->V);
    float* res = tmp.alloc<float>(3 * s->V);
    FEA_CUDA_TRY(cudaMemcpyAsync(nrm, normals, sizeof(float) * 3 * s->V, cudaMemcpyHostToDevice, s->stream));
    smooth_normals_dev(s, nrm, vertex_extrusion, face, res);
    FEA_CUDA_TRY(cudaMemcpyAsync(out, res, sizeof(float) * 3 * s->V, cudaMemcpyDeviceToHost, s->stream));
    FEA_CUDA_TRY(cudaStreamSynchronize(s->stream));
    API_END
}

int fea_smooth_normals_device(fea_solver* s, const float* normals, float vertex_extrusion, float* out) {
    API_BEGIN
    check_handle(s);
    if (!normals || !out) return fail(FEA_ERR_INVALID_ARGUMENT, "null normals or output");
    Scratch& tmp = s->scratch[2];
    tmp.rewind();
    smooth_normals_dev(s, normals, vertex_extrusion, tmp.alloc<float>(3 * s->T), out);
    FEA_CUDA_TRY(cudaStreamSynchronize(s->stream));
    API_END
}

int fea_ply_geometry(fea_solver* s, const float* normals, float vertex_extrusion, float threshold, int mesh_type,
                     float* positions, float* values, int64_t max_vertices, uint32_t* triangles,
                     int64_t max_triangles, int64_t* num_vertices, int64_t* num_triangles) {
    API_BEGIN
    check_handle(s);
    if (!normals || !num_vertices || !num_triangles) return fail(FEA_ERR_INVALID_ARGUMENT, "null argument");
    if (mesh_type < FEA_MESH_OPEN || mesh_type > FEA_MESH_MIRRORED) return fail(FEA_ERR_INVALID_ARGUMENT, "bad mesh type");
    PlyGeometry g;
    ply_geometry(s, normals, vertex_extrusion, threshold, mesh_type, g);
    const int64_t nv = (int64_t)g.val.size(), nt = (int64_t)g.tri.size() / 3;
    *num_vertices = nv;
    *num_triangles = nt;
    if (positions && values && nv <= max_vertices) {
        memcpy(positions, g.pos.data(), sizeof(float) * 3 * nv);
        memcpy(values, g.val.data(), sizeof(float) * nv);
    }
    if (triangles && nt <= max_triangles) memcpy(triangles, g.tri.data(), sizeof(uint32_t) * 3 * nt);
    API_END
}

int fea_export_ply(fea_solver* s, const char* path, const float* normals, float vertex_extrusion, float threshold,
                   int mesh_type, const float* color_coeffs) {
    API_BEGIN
    check_handle(s);
    if (!path || !normals) return fail(FEA_ERR_INVALID_ARGUMENT, "null path or normals");
    if (mesh_type < FEA_MESH_OPEN || mesh_type > FEA_MESH_MIRRORED) return fail(FEA_ERR_INVALID_ARGUMENT, "bad mesh type");
    float gray[21] = {0.f};
    gray[3] = gray[4] = gray[5] = 1.0f;  // color = (t, t, t)
    PlyGeometry g;
    ply_geometry(s, normals, vertex_extrusion, threshold, mesh_type, g);
    write_ply(path, g, color_coeffs ? color_coeffs : gray);
    API_END
}

int fea_adjoint_gray_scott(fea_solver* s, const float* u0, const float* v0, const float* target_u,
                           const float* target_v, int64_t nsteps, int64_t checkpoint_every, double* loss,
                           float* grad_u0, float* grad_v0, double* grad_params) {
    API_BEGIN
    check_handle(s);
    if (!u0 || !v0 || nsteps < 1 || checkpoint_every < 1)
        return fail(FEA_ERR_INVALID_ARGUMENT, "adjoint needs u0, v0, nsteps >= 1 and checkpoint_every >= 1");
    if (s->precision == FEA_FP64)
        adjoint_gs_host<double>(s, u0, v0, target_u, target_v, nsteps, checkpoint_every, loss, grad_u0, grad_v0,
                                grad_params);
    else
        adjoint_gs_host<float>(s, u0, v0, target_u, target_v, nsteps, checkpoint_every, loss, grad_u0, grad_v0,
                               grad_params);
    API_END
}

int fea_adjoint_gray_scott_device(fea_solver* s, const void* u0, const void* v0, const void* target_u,
                                  const void* target_v, int64_t nsteps, int64_t checkpoint_every, double* loss,
                                  void* grad_u0, void* grad_v0, double* grad_params) {
    API_BEGIN
    check_handle(s);
    if (!u0 || !v0 || nsteps < 1 || checkpoint_every < 1)
        return fail(FEA_ERR_INVALID_ARGUMENT, "adjoint needs u0, v0, nsteps >= 1 and checkpoint_every >= 1");
    if (s->precision == FEA_FP64)
        adjoint_gs_device<double>(s, u0, v0, target_u, target_v, nsteps, checkpoint_every, loss, grad_u0, grad_v0,
                                  grad_params);
    else
        adjoint_gs_device<float>(s, u0, v0, target_u, target_v, nsteps, checkpoint_every, loss, grad_u0, grad_v0,
                                 grad_params);
    API_END
}

int fea_clear_values(fea_solver* s) {
    API_BEGIN
    check_handle(s);
    Fields& F = s->F;
    const size_t n = rsize(s) * (size_t)(s->N > 0 ? s->N : 1);
    for (void* p : {F.u, F.v, F.a}) FEA_CUDA_TRY(cudaMemsetAsync(p, 0, n, s->stream));
    FEA_CUDA_TRY(cudaMemsetAsync(F.uv, 0, 2 * n, s->stream));
    FEA_CUDA_TRY(cudaMemsetAsync(&s->d_run->flags, 0, kCallFlagBytes, s->stream));
    s->acc_valid = false;
    invalidate_guess(s);
    FEA_CUDA_TRY(cudaStreamSynchronize(s->stream));
    API_END
}

int fea_set_values(fea_solver* s, const float* values) {
    API_BEGIN
    check_handle(s);
    if (!values) return fail(FEA_ERR_INVALID_ARGUMENT, "null values");
    if (s->precision == FEA_FP64) set_node_field<double>(s, values, displayed_field(s->prm));
    else set_node_field<float>(s, values, displayed_field(s->prm));
    if (displayed_field(s->prm) == 0) s->acc_valid = false;
    API_END
}

int fea_get_values(fea_solver* s, float* values) {
    API_BEGIN
    check_handle(s);
    if (!values) return fail(FEA_ERR_INVALID_ARGUMENT, "null values");
    if (s->precision == FEA_FP64) get_node_field<double>(s, values, displayed_field(s->prm));
    else get_node_field<float>(s, values, displayed_field(s->prm));
    API_END
}

int fea_set_fields(fea_solver* s, const float* u, const float* v) {
    API_BEGIN
    check_handle(s);
    if (s->precision == FEA_FP64) {
        if (u) set_node_field<double>(s, u, 0);
        if (v) set_node_field<double>(s, v, 1);
    } else {
        if (u) set_node_field<float>(s, u, 0);
        if (v) set_node_field<float>(s, v, 1);
    }
    s->acc_valid = false;
    API_END
}

int fea_get_fields(fea_solver* s, float* u, float* v) {
    API_BEGIN
    check_handle(s);
    if (s->precision == FEA_FP64) {
        if (u) get_node_field<double>(s, u, 0);
        if (v) get_node_field<double>(s, v, 1);
    } else {
        if (u) get_node_field<float>(s, u, 0);
        if (v) get_node_field<float>(s, v, 1);
    }
    API_END
}

int fea_set_fields_device(fea_solver* s, const void* u, const void* v) {
    API_BEGIN
    check_handle(s);
    if (s->precision == FEA_FP64) {
        if (u) copy_field_device<double>(s, u, nullptr, 0, true);
        if (v) copy_field_device<double>(s, v, nullptr, 1, true);
    } else {
        if (u) copy_field_device<float>(s, u, nullptr, 0, true);
        if (v) copy_field_device<float>(s, v, nullptr, 1, true);
    }
    s->acc_valid = false;
    FEA_CUDA_TRY(cudaStreamSynchronize(s->stream));
    API_END
}

int fea_get_fields_device(fea_solver* s, void* u, void* v) {
    API_BEGIN
    check_handle(s);
    if (s->precision == FEA_FP64) {
        if (u) copy_field_device<double>(s, nullptr, u, 0, false);
        if (v) copy_field_device<double>(s, nullptr, v, 1, false);
    } else {
        if (u) copy_field_device<float>(s, nullptr, u, 0, false);
        if (v) copy_field_device<float>(s, nullptr, v, 1, false);
    }
    FEA_CUDA_TRY(cudaStreamSynchronize(s->stream));
    API_END
}

int fea_advance_time(fea_solver* s, int64_t nsteps) {
    API_BEGIN
    check_handle(s);
    if (nsteps < 0) return fail(FEA_ERR_INVALID_ARGUMENT, "negative step count");
    if (nsteps == 0 || s->N == 0) return FEA_OK;
    if (s->precision == FEA_FP64) advance<double>(s, nsteps);
    else advance<float>(s, nsteps);
    API_END
}

int fea_synchronize(fea_solver* s) {
    API_BEGIN
    check_handle(s);
    FEA_CUDA_TRY(cudaStreamSynchronize(s->stream));
    API_END
}

int fea_get_status(fea_solver* s, fea_status* out) {
    API_BEGIN
    check_handle(s);
    if (!out) return fail(FEA_ERR_INVALID_ARGUMENT, "null status");
    FEA_CUDA_TRY(cudaMemcpyAsync(s->h_run, s->d_run, sizeof(RunState), cudaMemcpyDeviceToHost, s->stream));
    FEA_CUDA_TRY(cudaStreamSynchronize(s->stream));
    const RunState& r = *s->h_run;
    out->flags = r.flags | (r.expired ? FEA_STATUS_BREAKDOWN : 0u);
    out->last_iterations[0] = r.last_iters[0];
    out->last_iterations[1] = r.last_iters[1];
    out->last_rel_residual[0] = r.last_rel[0];
    out->last_rel_residual[1] = r.last_rel[1];
    out->steps_done = r.lost > 0 ? std::min<int64_t>(r.steps_done, s->run_steps - r.lost) : r.steps_done;
    out->total_iterations = r.total_iters;
    out->cg_launches = r.cg_launches;
    API_END
}

int fea_has_numerical_instability(fea_solver* s, int* out) {
    fea_status st;
    int rc = fea_get_status(s, &st);
    if (rc != FEA_OK) return rc;
    if (out) *out = (st.flags & (FEA_STATUS_BLOWUP | FEA_STATUS_NONFINITE)) ? 1 : 0;
    return FEA_OK;
}

int fea_get_info(fea_solver* s, fea_info* out) {
    API_BEGIN
    check_handle(s);
    if (!out) return fail(FEA_ERR_INVALID_ARGUMENT, "null info");
    out->num_vertices = s->V;
    out->num_triangles = s->T;
    out->num_boundary_points = s->nb;
    out->num_unknowns = s->N;
    out->nnz = s->P.nnz;
    out->max_row_nonzeros = s->P.max_row;
    out->precision = s->precision;
    out->boundary_condition = s->bc;
    out->rows_per_warp_lanes = s->lanes;
    out->device_bytes = s->mesh_mem.bytes + s->mat_mem.bytes + s->run_mem.bytes;
    for (const Scratch& k : s->scratch) out->device_bytes += k.bytes();
    API_END
}

int fea_get_matrix(fea_solver* s, int which, int32_t* row_ptr, int32_t* col, void* values, uint8_t* present) {
    API_BEGIN
    check_handle(s);
    const void* src = which == FEA_MATRIX_STIFFNESS ? s->K : which == FEA_MATRIX_MASS ? s->M
                    : which == FEA_MATRIX_ADVECTION ? s->Adv : nullptr;
    if (!src) return fail(FEA_ERR_INVALID_ARGUMENT, "bad matrix selector");
    FEA_CUDA_TRY(cudaStreamSynchronize(s->stream));
    if (row_ptr)
        FEA_CUDA_TRY(cudaMemcpy(row_ptr, s->P.row_ptr, sizeof(int32_t) * (s->N + 1), cudaMemcpyDeviceToHost));
    if (col && s->P.nnz) FEA_CUDA_TRY(cudaMemcpy(col, s->P.col, sizeof(int32_t) * s->P.nnz, cudaMemcpyDeviceToHost));
    if (values && s->P.nnz) FEA_CUDA_TRY(cudaMemcpy(values, src, rsize(s) * s->P.nnz, cudaMemcpyDeviceToHost));
    if (present && s->P.nnz) {
        if (which == FEA_MATRIX_ADVECTION)
            FEA_CUDA_TRY(cudaMemcpy(present, s->adv_present, s->P.nnz, cudaMemcpyDeviceToHost));
        else
            memset(present, 1, s->P.nnz);
    }
    API_END
}

int fea_get_idx_map(fea_solver* s, int32_t* idx_map, uint8_t* on_boundary) {
    API_BEGIN
    check_handle(s);
    FEA_CUDA_TRY(cudaStreamSynchronize(s->stream));
    if (idx_map) FEA_CUDA_TRY(cudaMemcpy(idx_map, s->idx, sizeof(int32_t) * s->V, cudaMemcpyDeviceToHost));
    if (on_boundary) FEA_CUDA_TRY(cudaMemcpy(on_boundary, s->ob, s->V, cudaMemcpyDeviceToHost));
    API_END
}

// Whether CG variant l runs on this handle: FEA_OK, FEA_ERR_INVALID_ARGUMENT
// (no such variant) or FEA_ERR_UNSUPPORTED (its layout or shared memory does
// not fit this mesh).
static int variant_check(const fea_solver* s, int l) {
    const bool csr = l == 4 || l == 8 || l == 16;
    const int stages = (l == 2 || l == 6 || l == 10) ? 2 : (l == 3 || l == 7 || l == 11) ? 3 : 0;
    const int ring = ring_stages(l);
    if (!csr && l != 0 && l != 1 && l != 13 && stages == 0 && ring == 0) return FEA_ERR_INVALID_ARGUMENT;
    if (!csr && !s->ell.ok) return FEA_ERR_UNSUPPORTED;
    if (s->stream_stages < stages) return FEA_ERR_UNSUPPORTED;
    if (ring && !ring_fits(s, s->ell, ring)) return FEA_ERR_UNSUPPORTED;
    return FEA_OK;
}

// The handle's variant while it lives.
struct VariantFor {
    fea_solver* s;
    int was;
    VariantFor(fea_solver* h, int l) : s(h), was(h->lanes) { s->lanes = l; }
    ~VariantFor() { s->lanes = was; }
};

int fea_autotune(fea_solver* s) {
    API_BEGIN
    check_handle(s);
    if (s->N == 0) return FEA_OK;
    const int kind = step_kind(s->prm);
    if (kind < 0) return fail(FEA_ERR_INVALID_ARGUMENT, "bad equation");
    ensure_operator(s, kind);
    cudaEvent_t e0, e1;
    FEA_CUDA_TRY(cudaEventCreate(&e0));
    FEA_CUDA_TRY(cudaEventCreate(&e1));
    const int cand[14] = {0, 1, 2, 3, 6, 7, 10, 11, 13, 14, 15, 4, 8, 16};
    float best = 1e30f;
    int best_l = s->lanes;
    for (int l : cand) {
        // on a mesh with stiff groups only the variants that use them: the others take
        // more iterations (170 against 68 a step on the 1024 x 1024 Gray-Scott grid),
        // which the time of one does not show
        if (variant_check(s, l) || (s->grp.n > 0 && !stiff_variant(s, l))) continue;
        const VariantFor probed(s, l);  // a variant's arguments are its own (which layout, deferred finish)
        probe_any(s, kind, l, true);
        for (int rep = 0; rep < 23; rep++) {
            if (rep == 3) FEA_CUDA_TRY(cudaEventRecord(e0, s->stream));
            probe_any(s, kind, l, false);
        }
        FEA_CUDA_TRY(cudaEventRecord(e1, s->stream));
        FEA_CUDA_TRY(cudaEventSynchronize(e1));
        float ms = 0;
        FEA_CUDA_TRY(cudaEventElapsedTime(&ms, e0, e1));
        if (ms < best) {
            best = ms;
            best_l = l;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    s->lanes = best_l;
    API_END
}

int fea_set_cg_variant(fea_solver* s, int variant) {
    API_BEGIN
    check_handle(s);
    switch (variant_check(s, variant)) {
    case FEA_ERR_INVALID_ARGUMENT:
        return fail(FEA_ERR_INVALID_ARGUMENT, "CG variant must be 0 to 4, 6 to 8, 10, 11 or 13 to 16");
    case FEA_ERR_UNSUPPORTED:
        return fail(FEA_ERR_UNSUPPORTED, s->ell.ok ? "streamed tiles exceed the shared memory on this mesh"
                                                   : "tile-ELL layout unavailable on this mesh");
    default: break;
    }
    s->lanes = variant;
    s->resident = false;  // an explicit choice names the kernels of the step graph
    API_END
}

int fea_get_stream(fea_solver* s, void** stream) {
    API_BEGIN
    check_handle(s);
    if (!stream) return fail(FEA_ERR_INVALID_ARGUMENT, "null stream output");
    *stream = (void*)s->stream;
    API_END
}

int fea_time_spmv(fea_solver* s, int reps, int flush_l2, double* ms_per_launch) {
    API_BEGIN
    check_handle(s);
    if (reps <= 0 || !ms_per_launch) return fail(FEA_ERR_INVALID_ARGUMENT, "bad arguments");
    if (s->N == 0) {
        *ms_per_launch = 0;
        return FEA_OK;
    }
    const int kind = step_kind(s->prm);
    if (kind < 0) return fail(FEA_ERR_INVALID_ARGUMENT, "bad equation");
    ensure_operator(s, kind);
    DeviceArena tmp;
    const size_t flush_bytes = (size_t)256 << 20;
    uint4* junk = nullptr;
    unsigned int* sink = nullptr;
    if (flush_l2) {
        junk = tmp.alloc<uint4>((int64_t)(flush_bytes / sizeof(uint4)));
        sink = tmp.alloc<unsigned int>(1);
        FEA_CUDA_TRY(cudaMemsetAsync(junk, 0, flush_bytes, s->stream));
    }
    auto flush = [&]() {
        if (!junk) return;
        k_read_flush<<<max_grid_blocks(), kBlock, 0, s->stream>>>(junk, (int64_t)(flush_bytes / sizeof(uint4)), sink);
        FEA_CHECK_LAUNCH();
    };
    flush();  // the memset's dirty lines leave the L2 before the first timing
    cudaEvent_t e0, e1;
    FEA_CUDA_TRY(cudaEventCreate(&e0));
    FEA_CUDA_TRY(cudaEventCreate(&e1));
    probe_any(s, kind, s->lanes, true);
    double total = 0;
    for (int rep = 0; rep < reps + 1; rep++) {  // the first launch is a warm-up
        flush();
        FEA_CUDA_TRY(cudaEventRecord(e0, s->stream));
        probe_any(s, kind, s->lanes, false);
        FEA_CUDA_TRY(cudaEventRecord(e1, s->stream));
        FEA_CUDA_TRY(cudaEventSynchronize(e1));
        float ms = 0;
        FEA_CUDA_TRY(cudaEventElapsedTime(&ms, e0, e1));
        if (rep > 0) total += ms;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    *ms_per_launch = total / reps;
    API_END
}

}  // extern "C"
