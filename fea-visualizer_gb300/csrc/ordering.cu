// ordering.cu -- the solver's ordering of the unknowns, computed on the device.
//
// Unknowns are sorted by the 63-bit Morton key of their points (coordinates
// quantised to 21 bits over the bounding box), ties by unknown number, then
// by stored-entry count within each tile of kTileRows rows.  Neighbouring
// points get nearby numbers, so a tile is a compact patch whose rows mostly
// reference each other, and the length order keeps the padding of the
// tile-ELL slices small.
//
// The sort is a stable least-significant-digit radix sort (8 passes of 8
// bits) of (key, unknown) pairs that start in unknown order.  Sorting on the
// host took 14.7 ms of the 57 ms of opening a 512 x 512 mesh; here it is under
// 1 ms, bound by the launches of its 24 small kernels.
#include "fea_internal.cuh"

namespace fea {
namespace {

constexpr int kSortItems = 16;  // elements per thread of a sort block
constexpr int kSortTile = kBlock * kSortItems;

// Floats as unsigned integers of the same order.
__device__ __forceinline__ uint32_t ordered_bits(float x) {
    const uint32_t b = __float_as_uint(x);
    return b & 0x80000000u ? ~b : b | 0x80000000u;
}
__device__ __forceinline__ float from_ordered(uint32_t b) {
    return __uint_as_float(b & 0x80000000u ? b & 0x7fffffffu : ~b);
}

// box[0..2]: smallest coordinates, box[3..5]: largest (ordered bits).
__global__ void k_bounds(const float* __restrict__ xyz, int64_t V, uint32_t* box) {
    __shared__ uint32_t lo[3], hi[3];
    if (threadIdx.x < 3) {
        lo[threadIdx.x] = 0xffffffffu;
        hi[threadIdx.x] = 0u;
    }
    __syncthreads();
    uint32_t l[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, h[3] = {0u, 0u, 0u};
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < V; i += (int64_t)gridDim.x * blockDim.x)
#pragma unroll
        for (int d = 0; d < 3; d++) {
            const uint32_t b = ordered_bits(xyz[3 * i + d]);
            l[d] = min(l[d], b);
            h[d] = max(h[d], b);
        }
#pragma unroll
    for (int d = 0; d < 3; d++) {
        l[d] = __reduce_min_sync(0xffffffffu, l[d]);
        h[d] = __reduce_max_sync(0xffffffffu, h[d]);
        if ((threadIdx.x & 31) == 0) {
            atomicMin(&lo[d], l[d]);
            atomicMax(&hi[d], h[d]);
        }
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        atomicMin(&box[threadIdx.x], lo[threadIdx.x]);
        atomicMax(&box[3 + threadIdx.x], hi[threadIdx.x]);
    }
}

__device__ __forceinline__ uint64_t spread3(uint32_t x) {  // 21 bits -> every third bit of 63
    uint64_t v = x & 0x1fffffu;
    v = (v | (v << 32)) & 0x1f00000000ffffull;
    v = (v | (v << 16)) & 0x1f0000ff0000ffull;
    v = (v | (v << 8)) & 0x100f00f00f00f00full;
    v = (v | (v << 4)) & 0x10c30c30c30c30c3ull;
    v = (v | (v << 2)) & 0x1249249249249249ull;
    return v;
}

__global__ void k_morton(const float* __restrict__ xyz, const int32_t* __restrict__ idx, int64_t V,
                         const uint32_t* __restrict__ box, uint64_t* key, int32_t* val) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < V; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t u = idx[i];
        if (u < 0) continue;
        uint64_t m = 0;
#pragma unroll
        for (int d = 0; d < 3; d++) {
            const double lo = from_ordered(box[d]), ext = (double)from_ordered(box[3 + d]) - lo;
            double t = ext > 0 ? __ddiv_rn((double)xyz[3 * i + d] - lo, ext) : 0.0;
            t = t < 0 ? 0 : (t > 1 ? 1 : t);
            m |= spread3((uint32_t)(t * 2097151.0)) << d;
        }
        key[u] = m;
        val[u] = u;
    }
}

__global__ void __launch_bounds__(kBlock) k_sort_hist(const uint64_t* __restrict__ key, int64_t n, int shift,
                                                      int32_t* hist) {
    __shared__ int32_t cnt[256];
    cnt[threadIdx.x] = 0;
    __syncthreads();
    const int64_t base = blockIdx.x * (int64_t)kSortTile + threadIdx.x;
#pragma unroll
    for (int k = 0; k < kSortItems; k++) {
        const int64_t i = base + (int64_t)k * kBlock;
        if (i < n) atomicAdd(&cnt[(key[i] >> shift) & 255], 1);
    }
    __syncthreads();
    hist[threadIdx.x * (int64_t)gridDim.x + blockIdx.x] = cnt[threadIdx.x];
}

// Exclusive scan of n counts in place by one block (each thread a contiguous
// run); n is 256 counts per sort block.
__global__ void __launch_bounds__(1024) k_sort_scan(int32_t* h, int64_t n) {
    __shared__ int32_t sm[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t per = ceil_div(n, 1024), b0 = min(n, threadIdx.x * per), b1 = min(n, b0 + per);
    int32_t sum = 0;
    for (int64_t i = b0; i < b1; i++) sum += h[i];
    int32_t s = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int32_t y = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += y;
    }
    if (lane == 31) sm[w] = s;
    __syncthreads();
    if (w == 0) {
        int32_t t = sm[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        sm[lane] = t;
    }
    __syncthreads();
    int32_t at = s - sum + (w > 0 ? sm[w - 1] : 0);
    for (int64_t i = b0; i < b1; i++) {
        const int32_t c = h[i];
        h[i] = at;
        at += c;
    }
}

// Stable scatter of one digit: the block's elements in rounds of kBlock; an
// element's place is the block's running offset of its digit (base[]), plus
// the digit's count in the round's earlier warps, plus its rank in its warp.
__device__ __forceinline__ void sort_scatter(const uint64_t* key, const int32_t* val, int64_t n, int shift,
                                             int32_t* base, uint64_t* key2, int32_t* val2) {
    __shared__ int32_t wc[kBlock / 32][256];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    for (int k = 0; k < kSortItems; k++) {
#pragma unroll
        for (int q = 0; q < kBlock / 32; q++) wc[q][t] = 0;
        __syncthreads();
        const int64_t i = blockIdx.x * (int64_t)kSortTile + (int64_t)k * kBlock + t;
        const bool in = i < n;
        const uint64_t x = in ? key[i] : 0;
        const unsigned d = in ? (unsigned)(x >> shift) & 255u : 256u;
        const unsigned same = __match_any_sync(0xffffffffu, d);
        const int rank = __popc(same & ((1u << lane) - 1u));
        if (in && rank == 0) wc[w][d] = __popc(same);
        __syncthreads();
        if (in) {
            int32_t at = base[d] + rank;
            for (int q = 0; q < w; q++) at += wc[q][d];
            key2[at] = x;
            val2[at] = val[i];
        }
        __syncthreads();
        int32_t add = 0;
#pragma unroll
        for (int q = 0; q < kBlock / 32; q++) add += wc[q][t];
        base[t] += add;
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kBlock) k_sort_scatter(const uint64_t* __restrict__ key,
                                                         const int32_t* __restrict__ val, int64_t n, int shift,
                                                         const int32_t* __restrict__ hist, uint64_t* key2,
                                                         int32_t* val2) {
    __shared__ int32_t base[256];
    base[threadIdx.x] = hist[threadIdx.x * (int64_t)gridDim.x + blockIdx.x];
    sort_scatter(key, val, n, shift, base, key2, val2);
}

// All passes of a sort that fits one block (n <= kSortTile): 8 launches of
// three kernels would cost more than the work.  key and val hold two halves
// of n; the sorted values end in the first.
__global__ void __launch_bounds__(kBlock) k_sort_small(uint64_t* key, int32_t* val, int n) {
    __shared__ int32_t base[256];
    __shared__ int32_t sm[kBlock / 32];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    for (int pass = 0; pass < 8; pass++) {
        const int from = (pass & 1) * n, to = n - from;
        base[t] = 0;
        __syncthreads();
        for (int i = t; i < n; i += kBlock) atomicAdd(&base[(key[from + i] >> (8 * pass)) & 255], 1);
        __syncthreads();
        const int32_t c = base[t];
        int32_t s = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        if (lane == 31) sm[w] = s;
        __syncthreads();
        for (int q = 0; q < w; q++) s += sm[q];
        base[t] = s - c;
        sort_scatter(key + from, val + from, n, 8 * pass, base, key + to, val + to);  // barrier before its first use
        __threadfence_block();
        __syncthreads();
    }
}

// Within each tile, rows by stored-entry count (stable).
__global__ void __launch_bounds__(kTileRows) k_tile_by_length(const int32_t* __restrict__ order,
                                                              const int32_t* __restrict__ rp, int64_t N, int32_t* inv,
                                                              int32_t* pos) {
    __shared__ int32_t len[kTileRows];
    const int t = threadIdx.x;
    const int64_t i = blockIdx.x * (int64_t)kTileRows + t;
    const int32_t u = i < N ? order[i] : -1;
    const int32_t l = u >= 0 ? rp[u + 1] - rp[u] : INT32_MAX;
    len[t] = l;
    __syncthreads();
    if (u < 0) return;
    int rank = 0;
    for (int q = 0; q < kTileRows; q++) rank += len[q] < l || (len[q] == l && q < t);
    const int64_t at = blockIdx.x * (int64_t)kTileRows + rank;
    inv[at] = u;
    pos[u] = (int32_t)at;
}

}  // namespace

void solver_order(const float* xyz, const int32_t* idx, int64_t V, const int32_t* rp, int64_t N, int32_t* inv,
                  int32_t* pos, cudaStream_t st) {
    if (N <= 0) return;
    const int nb = (int)ceil_div(N, kSortTile);
    DeviceArena tmp;
    // one allocation: keys, values, counts, bounding box
    uint64_t* key = tmp.alloc<uint64_t>(3 * N + 128 * (int64_t)nb + 3);
    int32_t* val = (int32_t*)(key + 2 * N);
    int32_t* hist = val + 2 * N;
    uint32_t* box = (uint32_t*)(hist + 256 * (int64_t)nb);
    FEA_CUDA_TRY(cudaMemsetAsync(box, 0xff, 3 * sizeof(uint32_t), st));
    FEA_CUDA_TRY(cudaMemsetAsync(box + 3, 0, 3 * sizeof(uint32_t), st));
    k_bounds<<<launch_grid(V), kBlock, 0, st>>>(xyz, V, box);
    FEA_CHECK_LAUNCH();
    k_morton<<<launch_grid(V), kBlock, 0, st>>>(xyz, idx, V, box, key, val);
    FEA_CHECK_LAUNCH();
    if (nb == 1) {
        k_sort_small<<<1, kBlock, 0, st>>>(key, val, (int)N);
        FEA_CHECK_LAUNCH();
    }
    for (int pass = 0; nb > 1 && pass < 8; pass++) {
        const int64_t from = (pass & 1) * N, to = N - from;
        k_sort_hist<<<nb, kBlock, 0, st>>>(key + from, N, 8 * pass, hist);
        FEA_CHECK_LAUNCH();
        k_sort_scan<<<1, 1024, 0, st>>>(hist, 256 * (int64_t)nb);
        FEA_CHECK_LAUNCH();
        k_sort_scatter<<<nb, kBlock, 0, st>>>(key + from, val + from, N, 8 * pass, hist, key + to, val + to);
        FEA_CHECK_LAUNCH();
    }
    k_tile_by_length<<<(int)ceil_div(N, kTileRows), kTileRows, 0, st>>>(val, rp, N, inv, pos);
    FEA_CHECK_LAUNCH();
    FEA_CUDA_TRY(cudaStreamSynchronize(st));  // the scratch is freed on return
}

}  // namespace fea
