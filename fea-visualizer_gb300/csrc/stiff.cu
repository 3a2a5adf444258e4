// stiff.cu -- stiff groups: an orthogonal change of basis on the few unknowns
// that nearly degenerate triangles tie together, for the ring CG kernels.
//
// A triangle whose corners are almost collinear adds (1 / area) q q^T to the
// stiffness matrix: one direction of its three unknowns becomes thousands of
// times stiffer than the rest.  The diagonal preconditioner scales all three
// unknowns down by that stiffness, which leaves the other two directions
// with eigenvalues near zero, and CG spends dozens of iterations on a
// handful of such triangles (jittered grids hold about one per thousand
// vertices).  The unknowns joined by a coupling |K_ij| > 0.75 sqrt(K_ii K_jj)
// form groups of up to four, strongest couplings first, and the iteration
// runs in the basis of each group's eigenvectors: A' = Q^T A Q, r' = Q^T r,
// x' = Q^T x, with Q the identity outside the groups.  Inside a group A' is
// diagonal, so the diagonal preconditioner of A' is the exact inverse of the
// group's block of A, while Q's orthogonality keeps |r| and |b|, hence the
// stopping test.  The kernels stay as they are: they get A' (a few entries
// of the diagonal-free tile-ELL layout change), its inverse diagonal, and
// the start values of the groups' rows.
//
// 0.75: on the 512 x 512 analog of the Gray-Scott workload (FP64 simulation)
// the first field took 60 CG iterations per solve without groups and 31 / 29
// / 28 / 27 with the bound at 0.8 / 0.75 / 0.7 / 0.6, the second 88 against
// 38 / 37 / 36 / 34; the unknowns in groups grow from 0.04% to 0.9%, and each
// one widens its neighbours' rows.  A uniformly stretched grid stays below
// 0.6, so anisotropic meshes are left alone.  Groups of more than four
// changed no iteration count.  On the GPU, 10 steps of the 1024 x 1024 Gray-
// Scott workload (about 800 unknowns of 1,048,576 in groups) take 19.9 ms
// against 46.4 ms without groups, the FP64 advection-diffusion adjoint of the 512
// x 512 grid 65.5 against 145 ms (both with this library's other changes of then).
#include <algorithm>
#include <array>
#include <unordered_map>

#include "cg_device.cuh"

namespace fea {
namespace {

constexpr double kStiffBound = 0.75;
// Meshes with fewer groups keep the diagonal iteration, whose loop stops at the
// tolerance itself.  Gray-Scott on jittered grids, resident launch, groups against
// none (iterations a step): 251 x 251, 22 groups, 20 steps 6.73 against 6.09 ms (65
// / 62); 330 x 330, 21 groups, 10 steps 4.64 against 5.45 (74 / 92); 500 x 500, 89
// groups, 8 steps 6.81 against 13.39 (75 / 177).  On the step graph 10.06 against
// 9.61, 6.79 against 8.01, 7.22 against 15.22.  Some 20 groups may go either way.
constexpr int kFewestGroups = 32;
// Smaller meshes are not searched: their solves are bound by launches, and the
// search would add a tenth of a millisecond to opening them.
constexpr int64_t kFewestRows = 4096;

struct StiffPair {
    float strength;
    int32_t i, j;
};

__global__ void k_diag_of(int64_t N, const int32_t* __restrict__ rp, const int32_t* __restrict__ col,
                          const double* __restrict__ K, double* d) {
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < N; r += (int64_t)gridDim.x * blockDim.x) {
        double v = 0;
        for (int32_t e = rp[r]; e < rp[r + 1]; e++)
            if (col[e] == r) v = K[e];
        d[r] = v;
    }
}

__global__ void k_stiff_pairs(int64_t N, const int32_t* __restrict__ rp, const int32_t* __restrict__ col,
                              const double* __restrict__ K, const double* __restrict__ d, int cap, StiffPair* out,
                              int* count) {
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < N; r += (int64_t)gridDim.x * blockDim.x)
        for (int32_t e = rp[r]; e < rp[r + 1]; e++) {
            const int32_t c = col[e];
            if (c <= r) continue;
            const double k2 = K[e] * K[e], dd = d[r] * d[c];
            if (!(dd > 0) || !(k2 > kStiffBound * kStiffBound * dd) || !isfinite(k2)) continue;
            const int at = atomicAdd(count, 1);
            if (at < cap) out[at] = {(float)(k2 / dd), (int32_t)r, c};
        }
}

// Entry (i, j) of A in the solver order (0 when not stored).
template <typename R, int NF>
__device__ double entry(const int32_t* __restrict__ rp, const int32_t* __restrict__ col,
                        const FV<R, NF>* __restrict__ A, int i, int j, int f) {
    int lo = rp[i], hi = rp[i + 1];
    while (lo < hi) {
        const int m = (lo + hi) >> 1;
        if (col[m] < j) lo = m + 1;
        else hi = m;
    }
    return lo < rp[i + 1] && col[lo] == j ? (double)A[lo].v[f] : 0.0;
}

// Eigenvectors of each group's block of A (its symmetric part), by cyclic
// Jacobi rotations (Golub and Van Loan, Matrix Computations, section 8.5);
// the rotations stop once the off-diagonal part is at round-off.  A block
// without a safely positive spectrum keeps the unit basis.  dinv holds the
// inverse diagonal of A on entry and that of A' on return.
template <typename R, int NF>
__global__ void k_stiff_basis(int n, const int32_t* __restrict__ mem, const int32_t* __restrict__ rp,
                              const int32_t* __restrict__ col, const FV<R, NF>* __restrict__ A, double* Q,
                              FV<R, NF>* dinv) {
    const int id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= n * NF) return;
    const int g = id / NF, f = id % NF;
    double a[4][4], q[4][4];
    int m[4];
#pragma unroll
    for (int i = 0; i < 4; i++) m[i] = mem[4 * g + i];
    double norm = 0;
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
            q[i][j] = i == j ? 1.0 : 0.0;
            a[i][j] = 0;
            if (m[i] >= 0 && m[j] >= 0)
                a[i][j] = 0.5 * (entry(rp, col, A, m[i], m[j], f) + entry(rp, col, A, m[j], m[i], f));
            norm = fmax(norm, fabs(a[i][j]));
        }
    for (int sweep = 0; sweep < 12; sweep++) {
        double off = 0;
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < i; j++) off = fmax(off, fabs(a[i][j]));
        if (!(off > 1e-17 * norm)) break;
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = i + 1; j < 4; j++) {
                if (a[i][j] == 0) continue;
                const double th = (a[j][j] - a[i][i]) / (2 * a[i][j]);
                const double t = (th >= 0 ? 1.0 : -1.0) / (fabs(th) + sqrt(th * th + 1));
                const double c = 1 / sqrt(t * t + 1), s = t * c;
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const double x = a[k][i], y = a[k][j];
                    a[k][i] = c * x - s * y;
                    a[k][j] = s * x + c * y;
                }
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const double x = a[i][k], y = a[j][k];
                    a[i][k] = c * x - s * y;
                    a[j][k] = s * x + c * y;
                    const double u = q[k][i], v = q[k][j];
                    q[k][i] = c * u - s * v;
                    q[k][j] = s * u + c * v;
                }
            }
    }
    bool ok = true;
#pragma unroll
    for (int i = 0; i < 4; i++)
        if (m[i] >= 0) ok = ok && a[i][i] > 1e-12 * norm && isfinite(a[i][i]);
#pragma unroll
    for (int i = 0; i < 4; i++) {
#pragma unroll
        for (int k = 0; k < 4; k++) Q[16 * (int64_t)id + 4 * i + k] = ok ? q[i][k] : i == k ? 1.0 : 0.0;
        if (ok && m[i] >= 0) dinv[m[i]].v[f] = (R)(1 / a[i][i]);
    }
}

// The entries of A' that differ from A's: (r, c) with r or c in a group.
template <typename R, int NF>
__global__ void k_stiff_entries(int nx, const int32_t* __restrict__ xr, const int32_t* __restrict__ xc,
                                const int32_t* __restrict__ mem, const int32_t* __restrict__ where,
                                const int32_t* __restrict__ rp, const int32_t* __restrict__ col,
                                const FV<R, NF>* __restrict__ A, const double* __restrict__ Q, FV<R, NF>* X) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nx; i += gridDim.x * blockDim.x) {
        const int r = xr[i], c = xc[i], wr = where[r], wc = where[c];
#pragma unroll
        for (int f = 0; f < NF; f++) {
            double sum = 0;
            for (int a = 0; a < (wr >= 0 ? 4 : 1); a++) {
                const int ra = wr >= 0 ? mem[(wr & ~3) + a] : r;
                if (ra < 0) continue;
                const double qa = wr >= 0 ? Q[16 * ((int64_t)(wr >> 2) * NF + f) + 4 * a + (wr & 3)] : 1.0;
                for (int b = 0; b < (wc >= 0 ? 4 : 1); b++) {
                    const int cb = wc >= 0 ? mem[(wc & ~3) + b] : c;
                    if (cb < 0) continue;
                    const double qb = wc >= 0 ? Q[16 * ((int64_t)(wc >> 2) * NF + f) + 4 * b + (wc & 3)] : 1.0;
                    sum += qa * qb * entry(rp, col, A, ra, cb, f);
                }
            }
            X[i].v[f] = (R)sum;
        }
    }
}

}  // namespace

bool stiff_groups_wanted(int64_t N) { return N >= kFewestRows; }

// Groups of unknowns of the pattern P by the stiffness matrix K, as arrays of
// four unknowns (-1 unused).  Deterministic: couplings in order of strength,
// then of index.
std::vector<std::array<int32_t, 4>> find_stiff_groups(const Pattern& P, const double* K, cudaStream_t st) {
    std::vector<std::array<int32_t, 4>> groups;
    const int64_t N = P.N;
    if (!stiff_groups_wanted(N) || P.nnz <= 0) return groups;
    const int cap = (int)(N / 16) + 64;
    DeviceArena tmp;
    double* d = tmp.alloc<double>(N);
    StiffPair* out = tmp.alloc<StiffPair>(cap);
    int* count = tmp.alloc<int>(1);
    FEA_CUDA_TRY(cudaMemsetAsync(count, 0, sizeof(int), st));
    k_diag_of<<<launch_grid(N), kBlock, 0, st>>>(N, P.row_ptr, P.col, K, d);
    FEA_CHECK_LAUNCH();
    k_stiff_pairs<<<launch_grid(N), kBlock, 0, st>>>(N, P.row_ptr, P.col, K, d, cap, out, count);
    FEA_CHECK_LAUNCH();
    int np = 0;
    FEA_CUDA_TRY(cudaMemcpyAsync(&np, count, sizeof(int), cudaMemcpyDeviceToHost, st));
    FEA_CUDA_TRY(cudaStreamSynchronize(st));
    // couplings this strong nearly everywhere: not a matter of a few triangles
    if (np == 0 || np > cap) return groups;
    std::vector<StiffPair> pairs(np);
    FEA_CUDA_TRY(cudaMemcpyAsync(pairs.data(), out, sizeof(StiffPair) * np, cudaMemcpyDeviceToHost, st));
    FEA_CUDA_TRY(cudaStreamSynchronize(st));
    std::sort(pairs.begin(), pairs.end(), [](const StiffPair& a, const StiffPair& b) {
        if (a.strength != b.strength) return a.strength > b.strength;
        return a.i != b.i ? a.i < b.i : a.j < b.j;
    });
    std::vector<int32_t> of(N, -1);  // group of an unknown
    std::vector<int> size;
    auto members = [&](int32_t u) { return of[u] < 0 ? 1 : size[of[u]]; };
    for (const StiffPair& p : pairs) {
        if ((of[p.i] >= 0 && of[p.i] == of[p.j]) || members(p.i) + members(p.j) > 4) continue;
        int32_t into = of[p.i] >= 0 ? of[p.i] : of[p.j];
        if (into < 0) {
            into = (int32_t)groups.size();
            groups.push_back({-1, -1, -1, -1});
            size.push_back(0);
        }
        for (int32_t u : {p.i, p.j}) {
            if (of[u] == into) continue;
            const int32_t from = of[u];
            std::array<int32_t, 4> add = {u, -1, -1, -1};
            if (from >= 0) {
                add = groups[from];
                groups[from] = {-1, -1, -1, -1};
                size[from] = 0;
            }
            for (int32_t w : add)
                if (w >= 0) {
                    groups[into][size[into]++] = w;
                    of[w] = into;
                }
        }
    }
    groups.erase(std::remove_if(groups.begin(), groups.end(), [](const std::array<int32_t, 4>& g) { return g[0] < 0; }),
                 groups.end());
    if ((int)groups.size() < kFewestGroups) groups.clear();
    return groups;
}

namespace {

// Entries of a row the plan takes: longer rows (hubs) leave a mesh without
// groups.
constexpr int kRowMost = 64;

// The columns of n rows (list[i], mapped through pos if given), kRowMost each
// (-1 past the end), with each row's number, first slot and length in head[3 i ..].
__global__ void k_copy_rows(int n, const int32_t* __restrict__ list, const int32_t* __restrict__ pos,
                            const int32_t* __restrict__ rp, const int32_t* __restrict__ col, int32_t* head,
                            int32_t* out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int32_t r = list[i] < 0 ? -1 : pos ? pos[list[i]] : list[i];
        const int32_t e0 = r < 0 ? 0 : rp[r], len = r < 0 ? 0 : rp[r + 1] - e0;
        head[3 * i] = r;
        head[3 * i + 1] = e0;
        head[3 * i + 2] = len;
        for (int k = 0; k < kRowMost; k++) out[(int64_t)i * kRowMost + k] = k < len ? col[e0 + k] : -1;
    }
}

__global__ void k_mark_rows(int n, const int32_t* __restrict__ list, int32_t* of) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        if (list[i] >= 0) of[list[i]] = i;
}

// Rows of the pattern copied to the host.
struct HostRows {
    std::vector<int32_t> head, col;
    HostRows(const std::vector<int32_t>& list, const int32_t* pos, const Pattern& Pc, cudaStream_t st)
        : head(3 * list.size()), col(kRowMost * list.size()) {
        const int n = (int)list.size();
        DeviceArena tmp;
        int32_t* d = tmp.alloc<int32_t>(n + 3 * (int64_t)n + kRowMost * (int64_t)n);
        FEA_CUDA_TRY(cudaMemcpyAsync(d, list.data(), sizeof(int32_t) * n, cudaMemcpyHostToDevice, st));
        k_copy_rows<<<launch_grid(n), kBlock, 0, st>>>(n, d, pos, Pc.row_ptr, Pc.col, d + n, d + 4 * (int64_t)n);
        FEA_CHECK_LAUNCH();
        FEA_CUDA_TRY(cudaMemcpyAsync(head.data(), d + n, sizeof(int32_t) * 3 * n, cudaMemcpyDeviceToHost, st));
        FEA_CUDA_TRY(cudaMemcpyAsync(col.data(), d + 4 * (int64_t)n, sizeof(int32_t) * kRowMost * n,
                                     cudaMemcpyDeviceToHost, st));
        FEA_CUDA_TRY(cudaStreamSynchronize(st));
    }
};

}  // namespace

bool plan_stiff_rows(const std::vector<std::array<int32_t, 4>>& unknowns, const Pattern& Pc, const int32_t* pos,
                     StiffGroups& G, ModRows& M, DeviceArena& keep, cudaStream_t st) {
    const int n = (int)unknowns.size();
    std::vector<int32_t> list;
    for (const auto& g : unknowns) list.insert(list.end(), g.begin(), g.end());
    const HostRows members(list, pos, Pc, st);
    // the groups in solver order, and the rows A' changes: every column of a
    // member's row (the pattern is symmetric; the diagonal is among them)
    std::vector<int32_t> mem(4 * n), rows;
    std::unordered_map<int32_t, int32_t> where;  // 4 * group + place
    for (int g = 0; g < n; g++) {
        int size = 0;
        for (int k = 0; k < 4; k++) {
            const int i = 4 * g + k;
            mem[i] = members.head[3 * i];
            if (mem[i] < 0) continue;
            size++;
            const int len = members.head[3 * i + 2];
            if (len > kRowMost) return false;
            rows.insert(rows.end(), members.col.begin() + i * kRowMost, members.col.begin() + i * kRowMost + len);
        }
        std::sort(mem.begin() + 4 * g, mem.begin() + 4 * g + size);  // unused places (-1) are last
        for (int k = 0; k < size; k++) where[mem[4 * g + k]] = 4 * g + k;
    }
    std::sort(rows.begin(), rows.end());
    rows.erase(std::unique(rows.begin(), rows.end()), rows.end());
    const HostRows old(rows, nullptr, Pc, st);
    std::unordered_map<int32_t, int32_t> at;  // row -> its place in `old`
    for (size_t i = 0; i < rows.size(); i++) at[rows[i]] = (int32_t)i;
    // the new rows: a column in a group brings the group's other members, a
    // group's row the columns of all its members; slots from nnz on are A's
    // entries that A' changes
    std::vector<int32_t> off(1, 0), col, slot, xr, xc;
    std::vector<std::pair<int32_t, int32_t>> row;  // column, slot (-1: changed)
    for (size_t i = 0; i < rows.size(); i++) {
        const int32_t r = rows[i];
        row.clear();
        auto add_row = [&](int32_t j, bool own) {
            const int32_t e0 = old.head[3 * j + 1], len = old.head[3 * j + 2];
            for (int k = 0; k < len; k++) {
                const int32_t c = old.col[(size_t)j * kRowMost + k];
                const auto w = where.find(c);
                if (w == where.end()) {
                    row.emplace_back(c, own ? e0 + k : -1);
                    continue;
                }
                for (int q = 0; q < 4; q++)
                    if (const int32_t m = mem[(w->second & ~3) + q]; m >= 0) row.emplace_back(m, -1);
            }
        };
        if (old.head[3 * i + 2] > kRowMost) return false;
        const auto w = where.find(r);
        if (w == where.end()) {
            add_row((int32_t)i, true);
        } else {
            for (int q = 0; q < 4; q++)
                if (const int32_t m = mem[(w->second & ~3) + q]; m >= 0) add_row(at[m], false);
        }
        std::sort(row.begin(), row.end());
        row.erase(std::unique(row.begin(), row.end()), row.end());
        for (const auto& e : row) {
            col.push_back(e.first);
            if (e.second < 0) {
                slot.push_back((int32_t)(Pc.nnz + xr.size()));
                xr.push_back(r);
                xc.push_back(e.first);
            } else {
                slot.push_back(e.second);
            }
        }
        off.push_back((int32_t)col.size());
    }
    if (Pc.nnz + (int64_t)xr.size() >= (int64_t)INT32_MAX) return false;
    auto upload = [&](const std::vector<int32_t>& v) {
        int32_t* d = keep.alloc<int32_t>((int64_t)v.size());
        FEA_CUDA_TRY(cudaMemcpyAsync(d, v.data(), sizeof(int32_t) * v.size(), cudaMemcpyHostToDevice, st));
        return d;
    };
    int32_t* of = keep.alloc<int32_t>(Pc.N);
    FEA_CUDA_TRY(cudaMemsetAsync(of, 0xff, sizeof(int32_t) * (size_t)Pc.N, st));
    int32_t* d_rows = upload(rows);
    k_mark_rows<<<launch_grid(rows.size()), kBlock, 0, st>>>((int)rows.size(), d_rows, of);
    FEA_CHECK_LAUNCH();
    M.of = of;
    M.off = upload(off);
    M.col = upload(col);
    M.slot = upload(slot);
    G.n = n;
    G.nx = (int)xr.size();
    G.mem = upload(mem);
    G.xr = upload(xr);
    G.xc = upload(xc);
    int32_t* wh = keep.alloc<int32_t>(Pc.N);
    FEA_CUDA_TRY(cudaMemsetAsync(wh, 0xff, sizeof(int32_t) * (size_t)Pc.N, st));
    k_mark_rows<<<launch_grid(4 * n), kBlock, 0, st>>>(4 * n, G.mem, wh);
    FEA_CHECK_LAUNCH();
    G.where = wh;
    FEA_CUDA_TRY(cudaStreamSynchronize(st));  // the host vectors go out of scope
    return true;
}

template <typename R, int NF>
void update_stiff_basis(const StiffGroups& G, const Pattern& Pc, const FV<R, NF>* A, const FV<R, NF>* dinv,
                        const StiffBasis& B, cudaStream_t st) {
    if (G.n == 0) return;
    FV<R, NF>* d = (FV<R, NF>*)B.dinv;
    FEA_CUDA_TRY(cudaMemcpyAsync(d, dinv, sizeof(FV<R, NF>) * (size_t)Pc.N, cudaMemcpyDeviceToDevice, st));
    k_stiff_basis<R, NF><<<(int)ceil_div((int64_t)G.n * NF, 64), 64, 0, st>>>(G.n, G.mem, Pc.row_ptr, Pc.col, A, B.Q, d);
    FEA_CHECK_LAUNCH();
    k_stiff_entries<R, NF><<<launch_grid(G.nx), kBlock, 0, st>>>(G.nx, G.xr, G.xc, G.mem, G.where, Pc.row_ptr, Pc.col,
                                                                 A, B.Q, (FV<R, NF>*)B.X);
    FEA_CHECK_LAUNCH();
}

#define FEA_INST_STIFF(R, NF)                                                                                  \
    template void update_stiff_basis<R, NF>(const StiffGroups&, const Pattern&, const FV<R, NF>*,              \
                                            const FV<R, NF>*, const StiffBasis&, cudaStream_t);
FEA_INST_STIFF(float, 1)
FEA_INST_STIFF(float, 2)
FEA_INST_STIFF(double, 1)
FEA_INST_STIFF(double, 2)

}  // namespace fea
