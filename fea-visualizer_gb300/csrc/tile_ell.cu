// tile_ell.cu -- the CG kernels' operator layout: tile-ELL with halo lists.
//
// The solver-order matrix is cut into tiles of kTileRows consecutive rows,
// each tile into 32-row slices.  A slice stores its rows' entries column by
// column (entry k of the slice's row `lane` at slice_off[s] + 32 k + lane),
// padded to the slice's longest row, so a warp reads one slice with fully
// coalesced loads and no row-pointer round trip.  Column indices are 16-bit
// and local to the tile: c - tile0 for rows of the tile, kTileRows + h for the
// tile's h-th halo column (the sorted distinct columns outside the tile).  The
// CG kernels place the vector they multiply for the tile's rows and its halo
// in shared memory, so every gathered operand is a shared-memory load.
// Entries keep their CSR order within a row (same summation order), and
// padding entries hold 0 with the row's own local index.  The diagonal-free
// variant of the layout leaves each row's diagonal entry out.
//
// The layout is built on the device, one block per tile: slice widths, then
// each tile's halo as a hash set of its outside columns (counted first, then
// sorted and written), then columns and slots.  The host build it replaces
// took 15.8 + 21.6 ms (full and diagonal-free) of the 57 ms of opening a 512 x
// 512 mesh, one core walking every entry several times.
#include <algorithm>

#include "fea_internal.cuh"

namespace fea {
namespace {

template <typename R, int NF>
__global__ void k_fill_tile_ell(int64_t E, const int32_t* __restrict__ emap, const FV<R, NF>* __restrict__ A,
                                const FV<R, NF>* __restrict__ X, int64_t nnz, FV<R, NF>* As) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < E; k += (int64_t)gridDim.x * blockDim.x) {
        const int32_t e = emap[k];
        FV<R, NF> v;
#pragma unroll
        for (int f = 0; f < NF; f++) v.v[f] = 0;
        if (e >= 0) v = e < nnz ? A[e] : X[e - nnz];
        As[k] = v;
    }
}

// Distinct halo columns a tile's hash set takes, at three quarters of its
// slots: meshes stay far below the first (a 512 x 512 jittered grid has at most
// 137), the second is above what any operand budget allows.
constexpr int kHaloSlots = 1024;
constexpr int kHaloSlotsMax = 16384;

// A row's entries: the pattern's, or the given ones (ModRows).
struct RowEntries {
    const int32_t *col, *slot;  // slot null: entry e has slot first + e
    int32_t first, n;
};
__device__ __forceinline__ RowEntries row_entries(const int32_t* rp, const int32_t* col, const ModRows& m, int64_t r) {
    const int32_t k = m.of ? m.of[r] : -1;
    if (k >= 0) return {m.col + m.off[k], m.slot + m.off[k], 0, m.off[k + 1] - m.off[k]};
    return {col + rp[r], nullptr, rp[r], rp[r + 1] - rp[r]};
}

struct EllTotals {
    unsigned long long entries;
    int hmax, emax, overflow;
};

// Entries per slice (32 x its longest row) and per tile, one block per tile.
__global__ void __launch_bounds__(kTileRows) k_slice_widths(const int32_t* __restrict__ rp,
                                                            const int32_t* __restrict__ col, ModRows mod, int64_t N,
                                                            bool skip_diag, int32_t* width, EllTotals* tot) {
    __shared__ unsigned long long sum;
    if (threadIdx.x == 0) sum = 0;
    __syncthreads();
    const int64_t r = blockIdx.x * (int64_t)kTileRows + threadIdx.x;
    int32_t len = 0;
    if (r < N) {
        const RowEntries row = row_entries(rp, col, mod, r);
        len = row.n;
        if (skip_diag)
            for (int32_t e = 0; e < row.n; e++) len -= row.col[e] == r;
    }
    const int32_t w = __reduce_max_sync(0xffffffffu, len);
    if ((threadIdx.x & 31) == 0) {
        width[blockIdx.x * (kTileRows / 32) + (threadIdx.x >> 5)] = 32 * w;
        atomicAdd(&sum, 32ull * (unsigned)w);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        atomicAdd(&tot->entries, sum);
        atomicMax(&tot->emax, (int)min(sum, (unsigned long long)INT32_MAX));
    }
}

// The tile's columns outside it, as a hash set in shared memory (open
// addressing, INT32_MAX empty).  Returns their number, or -1 past three
// quarters of the slots.  Every thread of the block calls it.
__device__ int halo_set(const int32_t* __restrict__ rp, const int32_t* __restrict__ col, const ModRows& mod, int64_t N,
                        int slots, int32_t* set) {
    __shared__ int count;
    const int64_t t0 = blockIdx.x * (int64_t)kTileRows, t1 = min(N, t0 + kTileRows);
    for (int i = threadIdx.x; i < slots; i += kTileRows) set[i] = INT32_MAX;
    if (threadIdx.x == 0) count = 0;
    __syncthreads();
    const int most = slots / 4 * 3;
    auto add = [&](int32_t c) {
        if (c >= t0 && c < t1) return;
        unsigned at = ((unsigned)c * 2654435761u >> 8) & (unsigned)(slots - 1);
        while (*(volatile int*)&count <= most) {
            const int32_t old = atomicCAS(&set[at], INT32_MAX, c);
            if (old == INT32_MAX) atomicAdd(&count, 1);
            if (old == INT32_MAX || old == c) break;
            at = (at + 1) & (unsigned)(slots - 1);
        }
    };
    // every entry of the pattern (a row given anew holds its old columns too),
    // then the rows given anew
    const int32_t e1 = rp[t1];
    for (int32_t e = rp[t0] + threadIdx.x; e < e1; e += kTileRows) add(col[e]);
    const int64_t r = t0 + threadIdx.x;
    if (mod.of && r < t1 && mod.of[r] >= 0) {
        const RowEntries row = row_entries(rp, col, mod, r);
        for (int32_t e = 0; e < row.n; e++) add(row.col[e]);
    }
    __syncthreads();
    return count <= most ? count : -1;
}

__global__ void __launch_bounds__(kTileRows) k_halo_count(const int32_t* __restrict__ rp,
                                                          const int32_t* __restrict__ col, ModRows mod, int64_t N,
                                                          int slots, int32_t* hcnt, EllTotals* tot) {
    extern __shared__ int32_t set[];
    const int n = halo_set(rp, col, mod, N, slots, set);
    if (threadIdx.x == 0) {
        hcnt[blockIdx.x] = max(n, 0);
        if (n < 0) atomicExch(&tot->overflow, 1);
        else atomicMax(&tot->hmax, n);
    }
}

// Halo lists (sorted), local columns, column pairs and slots of one tile.
__global__ void __launch_bounds__(kTileRows) k_fill_pattern(const int32_t* __restrict__ rp,
                                                            const int32_t* __restrict__ col, ModRows mod, int64_t N,
                                                            bool skip_diag, int slots,
                                                            const int32_t* __restrict__ slice_off,
                                                            const int32_t* __restrict__ halo_off, int32_t* halo_col,
                                                            uint16_t* lcol, uint32_t* lcol2, int32_t* emap) {
    extern __shared__ int32_t set[];
    const int n = halo_set(rp, col, mod, N, slots, set);
    for (int size = 2; size <= slots; size <<= 1)  // bitonic sort; the empty slots go last
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int i = threadIdx.x; i < slots / 2; i += kTileRows) {
                const int lo = 2 * i - (i & (stride - 1)), hi = lo + stride;
                const int32_t a = set[lo], b = set[hi];
                if ((a > b) == ((lo & size) == 0)) {
                    set[lo] = b;
                    set[hi] = a;
                }
            }
            __syncthreads();
        }
    const int32_t h0 = halo_off[blockIdx.x];
    for (int i = threadIdx.x; i < n; i += kTileRows) halo_col[h0 + i] = set[i];
    const int64_t t0 = blockIdx.x * (int64_t)kTileRows, r = t0 + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const int64_t s = blockIdx.x * (int64_t)(kTileRows / 32) + (threadIdx.x >> 5);
    const int32_t sb = slice_off[s], w = (slice_off[s + 1] - sb) / 32;
    RowEntries row{};
    if (r < N) row = row_entries(rp, col, mod, r);
    int32_t e = 0;
    uint32_t first = 0;
    for (int32_t k = 0; k < w; k++) {
        if (skip_diag && e < row.n && row.col[e] == r) e++;
        uint32_t lc = (uint32_t)threadIdx.x;  // padding: the row's own slot, value 0
        int32_t slot = -1;
        if (e < row.n) {
            const int32_t c = row.col[e];
            if (c >= t0 && c < t0 + kTileRows) {
                lc = (uint32_t)(c - t0);
            } else {
                int lo = 0, hi = n;
                while (lo < hi) {
                    const int m = (lo + hi) >> 1;
                    if (set[m] < c) lo = m + 1;
                    else hi = m;
                }
                lc = (uint32_t)(kTileRows + lo);
            }
            slot = row.slot ? row.slot[e] : row.first + e;
            e++;
        }
        const int32_t at = sb + 32 * k + lane;
        lcol[at] = (uint16_t)lc;
        emap[at] = slot;
        if (lcol2) {
            if (k & 1) lcol2[sb + 32 * (k >> 1) + lane] = first | lc << 16;
            else if (k == w - 1) lcol2[sb + 32 * (k >> 1) + lane] = lc | lc << 16;
            first = lc;
        }
    }
}

}  // namespace

bool build_tile_ell(const int32_t* rp, const int32_t* col, int64_t N, size_t fv_bytes, size_t smem_budget, TileEll& L,
                    DeviceArena& keep, cudaStream_t st, bool skip_diag, const ModRows* given) {
    const ModRows mod = given ? *given : ModRows{};
    L = TileEll{};
    if (N <= 0) return false;
    const int64_t ntiles = ceil_div(N, kTileRows), nslices = ntiles * (kTileRows / 32);
    DeviceArena tmp;
    EllTotals* tot = (EllTotals*)tmp.alloc<unsigned char>(sizeof(EllTotals) + sizeof(int32_t) * (nslices + ntiles));
    int32_t* width = (int32_t*)(tot + 1);
    int32_t* hcnt = width + nslices;
    EllTotals h{};
    // 16-bit local indices and the shared-memory slice of the tile's operand
    const int64_t limit = std::min<int64_t>(65535, (int64_t)(smem_budget / fv_bytes)) - kTileRows;
    int slots = kHaloSlots;
    for (;;) {
        FEA_CUDA_TRY(cudaMemsetAsync(tot, 0, sizeof(EllTotals), st));
        k_slice_widths<<<(int)ntiles, kTileRows, 0, st>>>(rp, col, mod, N, skip_diag, width, tot);
        FEA_CHECK_LAUNCH();
        if (slots > kHaloSlots)
            FEA_CUDA_TRY(cudaFuncSetAttribute(k_halo_count, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * slots));
        k_halo_count<<<(int)ntiles, kTileRows, 4 * slots, st>>>(rp, col, mod, N, slots, hcnt, tot);
        FEA_CHECK_LAUNCH();
        FEA_CUDA_TRY(cudaMemcpyAsync(&h, tot, sizeof(h), cudaMemcpyDeviceToHost, st));
        FEA_CUDA_TRY(cudaStreamSynchronize(st));
        if (!h.overflow) break;
        if (slots == kHaloSlotsMax) return false;  // more distinct columns than any operand budget holds
        slots = kHaloSlotsMax;
    }
    if (h.entries >= (unsigned long long)INT32_MAX || h.hmax > limit) return false;
    const int64_t E = (int64_t)h.entries;
    L.E = E;
    L.ntiles = (int)ntiles;
    L.hmax = h.hmax;
    L.emax = h.emax;
    L.slice_off = keep.alloc<int32_t>(nslices + 1);
    L.halo_off = keep.alloc<int32_t>(ntiles + 1);
    exclusive_scan_i32(width, L.slice_off, nslices, st);
    const int64_t nh = exclusive_scan_i32(hcnt, L.halo_off, ntiles, st);
    L.halo_col = keep.alloc<int32_t>(std::max<int64_t>(1, nh));
    L.lcol = keep.alloc<uint16_t>(std::max<int64_t>(1, E));
    L.emap = keep.alloc<int32_t>(std::max<int64_t>(1, E));
    if (!skip_diag) {
        L.lcol2 = keep.alloc<uint32_t>(std::max<int64_t>(1, E));
        FEA_CUDA_TRY(cudaMemsetAsync(L.lcol2, 0, sizeof(uint32_t) * (size_t)std::max<int64_t>(1, E), st));
    }
    if (slots > kHaloSlots)
        FEA_CUDA_TRY(cudaFuncSetAttribute(k_fill_pattern, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * slots));
    k_fill_pattern<<<(int)ntiles, kTileRows, 4 * slots, st>>>(rp, col, mod, N, skip_diag, slots, L.slice_off, L.halo_off,
                                                              L.halo_col, L.lcol, L.lcol2, L.emap);
    FEA_CHECK_LAUNCH();
    L.ok = true;
    return true;
}

template <typename R, int NF>
void fill_tile_ell(const TileEll& L, const FV<R, NF>* A, FV<R, NF>* As, cudaStream_t st, const FV<R, NF>* X,
                   int64_t nnz) {
    if (!L.ok || L.E == 0) return;
    k_fill_tile_ell<R, NF><<<launch_grid(L.E), kBlock, 0, st>>>(L.E, L.emap, A, X, nnz, As);
    FEA_CHECK_LAUNCH();
}

template void fill_tile_ell<float, 1>(const TileEll&, const FV<float, 1>*, FV<float, 1>*, cudaStream_t, const FV<float, 1>*,
                                      int64_t);
template void fill_tile_ell<float, 2>(const TileEll&, const FV<float, 2>*, FV<float, 2>*, cudaStream_t, const FV<float, 2>*,
                                      int64_t);
template void fill_tile_ell<double, 1>(const TileEll&, const FV<double, 1>*, FV<double, 1>*, cudaStream_t, const FV<double, 1>*,
                                      int64_t);
template void fill_tile_ell<double, 2>(const TileEll&, const FV<double, 2>*, FV<double, 2>*, cudaStream_t, const FV<double, 2>*,
                                      int64_t);

}  // namespace fea
