// resident.cu -- the step loop of small and mid-size meshes in one kernel.
//
// The step graph (cg.cu) launches one kernel per CG iteration; on a mesh whose
// tiles all run at once such a launch costs 5 to 9 us whatever it computes,
// and a step's other passes and loop nodes another 50 to 120 us.  Here one
// launch runs every step: each block owns a run of 256-row tiles, keeps their
// diagonal-free tile-ELL operator (tile_ell.cu) in shared memory and its rows'
// CG vectors in registers for the whole launch.  The recurrences and the sums'
// precision are those of the ring kernels; of the CG scalars, beta g / alpha is
// taken as beta (g / alpha), with as many roundings.  Every block merges all
// blocks' partials in one fixed order and so computes the same scalars.
//
// What the blocks exchange carries its own arrival flag: every 4-byte word
// travels in an 8-byte store beside a 4-byte epoch, and the reader polls the
// word it needs until the epoch is the expected one.  So there are no grid
// barriers and no fences.  The buffers are safe to overwrite because a block
// can send partials of one reduction only after it has read everything of the
// one before: w alternates between two buffers, the partials too, x by the
// step's parity, and the others are rewritten only after a reduction that
// follows their last read.
//
// Reductions: up to 16 blocks run as one thread block cluster and write their
// partials into each other's shared memory; more blocks send them to block 0
// and poll its totals.  Clocks per reduction of six values (a loop of nothing
// else): 1,750 in a cluster of 16 against 3,430 through the L2; 128 blocks
// 5,120 through block 0 against 8,740 with every block reading every partial
// (the polls of all blocks meet on the same lines) and about 7,300 for a
// counter barrier and a second read.  In this kernel the every-block form took
// 11.1 ms against 6.3 (Gray-Scott, 251 x 251 grid, 124 blocks, 20 steps).
//
// Per iteration a block publishes only w' = A u' of its rows.  A halo slot's
// thread keeps its own copy of the halo row's r and s and advances them from
// that w exactly as the owner does (same operations, same operands), so u' of
// the halo costs one 8- to 32-byte load per slot.
//
// The blocks wait on one another, so several run as one cluster or as a
// cooperative launch.  Every wait is bounded; on expiry the launch raises
// FEA_STATUS_BREAKDOWN and leaves.
#include <algorithm>
#include <cstdlib>
#include <type_traits>

#include "cg_device.cuh"

namespace fea {
namespace {

constexpr int kResThreads = 512;  // two tiles of 256 rows at a time; 128 registers a thread
constexpr long long kWaitClocks = 6000000000ll;  // about 3 s of waiting at most (FEA_WAIT_CLOCKS: another bound)
constexpr int64_t kResidentSteps = 256;          // steps of one launch at most
constexpr int kMaxBlocks = 160;                  // slots per value of the partials' buffers
constexpr int kClusterBlocks = 16;               // blocks of a cluster launch (above 8: opt-in)
// Tiles per block up to which a mesh runs as one cluster.  Heat on a grid, 6
// steps, one cluster against a cooperative grid of one-tile blocks: FP32 16
// tiles 1,233 against 1,381 us, 27 tiles (two a block) 1,155 against 1,397;
// three a block lost (38 tiles 1,397 against 1,200).  FP64, bound by the SMs'
// FP64 rate: 16 tiles 2,650 against 3,060 us, two a block lost (20 tiles 2,865
// against 2,373, 413 iterations).
template <typename R>
constexpr int kClusterTiles = sizeof(R) == 4 ? 2 : 1;

// Lambdas hold the launch's registers by reference: out of line they would put
// them on the stack.
#define FEA_INLINE __attribute__((always_inline))

// A value the compiler cannot hoist out of a loop: the addresses of the dozens
// of arrays a step touches would otherwise be kept in registers through the
// iterations, which touch one.
__device__ __forceinline__ int opaque(int x) {
    asm volatile("" : "+r"(x));
    return x;
}

// ---- flagged words -----------------------------------------------------------------
// An element of T (4, 8, 16 bytes) as sizeof(T) / 4 pairs {word, epoch}.
template <typename T>
constexpr int kPairs = sizeof(T) / 4;

template <typename T>
__device__ __forceinline__ void put(uint2* buf, int64_t i, const T& v, uint32_t epoch) {
    constexpr int n = kPairs<T>;
    uint32_t w[n];
    memcpy(w, &v, sizeof(T));
    uint2* p = buf + i * n;
    if constexpr (n == 1) {
        asm volatile("st.volatile.global.v2.u32 [%0], {%1, %2};" ::"l"(p), "r"(w[0]), "r"(epoch) : "memory");
    } else {
#pragma unroll
        for (int k = 0; k < n; k += 2)
            asm volatile("st.volatile.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(p + k), "r"(w[k]), "r"(epoch),
                         "r"(w[k + 1]), "r"(epoch)
                         : "memory");
    }
}

// One try; false while a word has not arrived.
template <typename T>
__device__ __forceinline__ bool try_get(const uint2* buf, int64_t i, T& v, uint32_t epoch) {
    constexpr int n = kPairs<T>;
    uint32_t w[n];
    const uint2* p = buf + i * n;
    bool ok = true;
    if constexpr (n == 1) {
        uint32_t e;
        asm volatile("ld.volatile.global.v2.u32 {%0, %1}, [%2];" : "=r"(w[0]), "=r"(e) : "l"(p) : "memory");
        ok = e == epoch;
    } else {
#pragma unroll
        for (int k = 0; k < n; k += 2) {
            uint32_t e0, e1;
            asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(w[k]), "=r"(e0), "=r"(w[k + 1]), "=r"(e1)
                         : "l"(p + k)
                         : "memory");
            ok = ok && e0 == epoch && e1 == epoch;
        }
    }
    memcpy(&v, w, sizeof(T));
    return ok;
}

// How long a wait may last, and where a block notes that one expired.
struct Patience {
    volatile int* dead;
    long long most;
    __device__ __forceinline__ bool over(long long since) const {
        if (!*dead && clock64() - since <= most) return false;
        *dead = 1;
        return true;
    }
};

template <typename T>
__device__ __forceinline__ T get(const uint2* buf, int64_t i, uint32_t epoch, const Patience& wait) {
    T v;
    if (try_get(buf, i, v, epoch)) return v;
    const long long t0 = clock64();
    while (!try_get(buf, i, v, epoch))
        if (wait.over(t0)) break;
    return v;
}

// n values at once: every missing one is asked for before any is waited for, so
// a round of polls costs one trip through the L2.  One value after another,
// Gray-Scott on a 251 x 251 grid (124 blocks) took 7,640 us against 6,320, and
// heat on a 550 x 550 grid (four passes) 27,570 against 20,140.
template <int n, typename T, typename Want, typename Try>
__device__ __forceinline__ void get_all(T (&v)[n], Want want, Try attempt, const Patience& wait) {
    bool here[n];
#pragma unroll
    for (int i = 0; i < n; i++) here[i] = !want(i);
    long long t0 = 0;
    for (;;) {
        bool all = true;
        T x[n];
        bool ok[n];
#pragma unroll
        for (int i = 0; i < n; i++) ok[i] = here[i] || attempt(i, x[i]);
#pragma unroll
        for (int i = 0; i < n; i++) {
            if (!here[i]) v[i] = x[i];
            here[i] = ok[i];
            all = all && ok[i];
        }
        if (all) return;
        if (t0 == 0) t0 = clock64();
        if (wait.over(t0)) return;
    }
}

// An 8-byte value as two flagged words in the shared memory of block `rank` of
// the cluster, at the place of this block's p; and the wait for it.
__device__ __forceinline__ void put_remote(uint2* p, int rank, const uint2& v, uint32_t epoch) {
    uint32_t at;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                 : "=r"(at)
                 : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    asm volatile("st.relaxed.cluster.shared::cluster.v2.u32 [%0], {%1, %2};" ::"r"(at), "r"(v.x), "r"(epoch) : "memory");
    asm volatile("st.relaxed.cluster.shared::cluster.v2.u32 [%0], {%1, %2};" ::"r"(at + 8), "r"(v.y), "r"(epoch)
                 : "memory");
}
__device__ __forceinline__ uint2 get_shared(const uint2* p, uint32_t epoch, const Patience& wait) {
    const uint32_t at = (uint32_t)__cvta_generic_to_shared(p);
    uint2 v;
    uint32_t e0, e1;
    long long t0 = 0;
    for (;;) {
        asm volatile("ld.relaxed.cluster.shared::cta.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(e0) : "r"(at) : "memory");
        asm volatile("ld.relaxed.cluster.shared::cta.v2.u32 {%0, %1}, [%2];"
                     : "=r"(v.y), "=r"(e1)
                     : "r"(at + 8)
                     : "memory");
        if (e0 == epoch && e1 == epoch) return v;
        if (t0 == 0) t0 = clock64();
        if (wait.over(t0)) return v;
    }
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// ---- sums ------------------------------------------------------------------------------

// Warp sums of N accumulators by halving exchanges: with N padded to W = 2, 4 or
// 8 each lane ends with one value's sum (W - 1 + 5 - log2 W merges instead of 5 N),
// which the lanes with zero low bits store.
template <int N, typename A>
__device__ __forceinline__ void warp_scatter_sums(const A (&in)[N], typename A::Packed* out) {
    constexpr int W = N <= 2 ? 2 : N <= 4 ? 4 : 8;
    const int lane = threadIdx.x & 31;
    A v[W];
#pragma unroll
    for (int k = 0; k < N; k++) v[k] = in[k];
    int off = 16, slot = 0;
#pragma unroll
    for (int half = W / 2; half >= 1; half >>= 1) {
        const bool up = (lane & off) != 0;
        slot = 2 * slot + (up ? 1 : 0);
#pragma unroll
        for (int k = 0; k < half; k++) {
            A keep = up ? v[half + k] : v[k];
            const auto g = (up ? v[k] : v[half + k]).pack();
            typename A::Packed o;
            if constexpr (std::is_same_v<A, Acc<float>>) {
                o.x = __shfl_xor_sync(0xffffffffu, g.x, off);
                o.y = __shfl_xor_sync(0xffffffffu, g.y, off);
            } else {
                o = __shfl_xor_sync(0xffffffffu, g, off);
            }
            keep.merge(A::unpack(o));
            v[k] = keep;
        }
        off >>= 1;
    }
#pragma unroll
    for (int o = 16 / W; o > 0; o >>= 1) v[0].shfl_add(o);
    if ((lane & (32 / W - 1)) == 0 && slot < N) out[slot] = v[0].pack();
}

__device__ __forceinline__ FF from_lane(const FF& x, int lane) {
    FF y;
    y.hi = __shfl_sync(0xffffffffu, x.hi, lane);
    y.lo = __shfl_sync(0xffffffffu, x.lo, lane);
    return y;
}

// Lane 0's packed accumulator in every lane.
__device__ __forceinline__ float2 lane0(float2 v) {
    return make_float2(__shfl_sync(0xffffffffu, v.x, 0), __shfl_sync(0xffffffffu, v.y, 0));
}
__device__ __forceinline__ double lane0(double v) { return __shfl_sync(0xffffffffu, v, 0); }

// Everything a launch adds to the step's arguments.
template <typename R>
struct ResidentArgs {
    int kind, steps, first;  // equation kind; steps of this launch; the first launch of a call
    int T, tpb;              // tiles per block, tiles a block works on at a time
    int cluster;             // the blocks are one cluster
    int us;                  // staged operands per tile: kTileRows + the largest halo
    long long left;          // steps of the call from this launch's first on
    long long wait;          // clocks a wait may last
    const R* Ks;             // tile-ELL copies of K and Adv (M: StepArgs::Ms)
    const R* Advs;
    const int32_t* where;    // stiff groups: 4 * group + place of a row, -1 elsewhere
    uint2 *wl[2], *xl[2], *rl[2], *yl, *pl;  // flagged w, x, r, wave operand and the partials
};

// kP: tiles per thread group (a block's tile lt = q * tpb + group is pass q).
template <typename R, int NF, int kP>
__global__ void __launch_bounds__(kResThreads, 1) k_resident(StepArgs<R, NF> a, ResidentArgs<R> ra) {
    using V = FV<R, NF>;
    constexpr int NV = 3 * NF;
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ double red[kResThreads / 32][8];  // packed accumulators (8 bytes of either type)
    __shared__ double tot[8];
    __shared__ uint2 part[2][8][kClusterBlocks][2];  // a cluster's partials, by parity, value and block
    __shared__ CgState st;
    __shared__ struct {  // what an iteration needs of the state
        R alpha[NF], beta[NF];
        int act[NF], any;
    } ctl;
    __shared__ struct {  // the last completed step's solves
        int iters[NF];
        double rr[NF], bb[NF];
    } last;
    __shared__ unsigned int sflags;
    __shared__ int dead, sstop;
    const int grp = threadIdx.x >> 8, t = threadIdx.x & 255, lane = t & 31, w8 = t >> 5;
    const int j = (t & 7) * 32 + (t >> 3);  // halo slot, dealt round-robin over the warps
    const int us = ra.us, emx = a.emax_od, nb = (int)gridDim.x;
    V* const ent = reinterpret_cast<V*>(dyn);
    uint16_t* const lcs = reinterpret_cast<uint16_t*>(dyn + (((size_t)ra.T * emx * sizeof(V) + 15) & ~(size_t)15));
    V* const ub = reinterpret_cast<V*>(reinterpret_cast<unsigned char*>(lcs) + (((size_t)ra.T * emx * 2 + 15) & ~(size_t)15));
    RunState* const run = a.run;
    if (threadIdx.x == 0) {
        dead = 0;
        sflags = 0;
        sstop = ra.first ? 0 : run->halt;
    }
    __syncthreads();
    if (sstop) return;  // an earlier launch of this call stopped (the same value in every block)
    uint32_t epoch = run->epoch;  // of the last exchange; block 0 stores it when the launch ends
    if (ra.cluster) {  // no block writes into another before that one has cleared its slots
        for (int i = threadIdx.x; i < 2 * 8 * kClusterBlocks * 2; i += blockDim.x)
            (&part[0][0][0][0])[i] = make_uint2(0, epoch);
        cluster_barrier();
    }

    // the operator into shared memory, once per launch
    {
        const int ntiles = (int)ceil_div(a.N, kTileRows);
        for (int lt = 0; lt < ra.T; lt++) {
            const int tile = (int)blockIdx.x * ra.T + lt;
            if (tile >= ntiles) break;
            const int32_t e0 = a.slice_off_od[tile * 8], n = a.slice_off_od[tile * 8 + 8] - e0;
            for (int i = threadIdx.x; i < n; i += blockDim.x) {
                ent[lt * emx + i] = ldfv(a.As_od + e0 + i);
                lcs[lt * emx + i] = a.lcol_od[e0 + i];
            }
        }
    }
    // per pass: the thread's row (-1: none), the warp's slice, the halo column
    int rowq[kP], sref[kP], hcol[kP];
    V cd[kP], hd[kP];
#pragma unroll
    for (int q = 0; q < kP; q++) {
        const int lt = q * ra.tpb + grp, tile = (int)blockIdx.x * ra.T + lt, row = tile * kTileRows + t;
        const bool in = lt < ra.T && tile < (int)ceil_div(a.N, kTileRows);
        rowq[q] = in && row < a.N ? row : -1;
        sref[q] = 0;
        hcol[q] = -1;
        cd[q] = hd[q] = V{};
        if (in) {
            const int32_t e0 = a.slice_off_od[tile * 8], sb = a.slice_off_od[tile * 8 + w8] - e0;
            sref[q] = sb << 16 | (a.slice_off_od[tile * 8 + w8 + 1] - e0 - sb) >> 5;
            const int32_t h0 = a.halo_off_od[tile];
            if (j < a.halo_off_od[tile + 1] - h0) hcol[q] = a.halo_col_od[h0 + j];
            if (rowq[q] >= 0) cd[q] = ldfv(a.dinv_it + row);
            if (hcol[q] >= 0) hd[q] = ldfv(a.dinv_it + hcol[q]);
        }
    }
    const Patience wait{&dead, ra.wait};
    auto ub_of = [&](int q) FEA_INLINE { return ub + (q * ra.tpb + grp) * us; };
    // outside the iterations: the thread's row and tile, addresses not kept
    auto row_of = [&](int q) FEA_INLINE { return (int64_t)opaque(rowq[q]); };
    auto tile_of = [&](int q) FEA_INLINE {
        const int lt = q * opaque(ra.tpb) + grp, tile = (int)blockIdx.x * ra.T + lt;
        return lt < ra.T && tile < (int)ceil_div(a.N, kTileRows) ? tile : -1;
    };

    int ph = 0;  // parity of the partials' buffers
    // Totals of the blocks' accumulators into tot[], in every block.  False when
    // a wait expired.
    auto reduce = [&](auto& acc) FEA_INLINE {
        using A = std::remove_reference_t<decltype(acc[0])>;
        using Pk = typename A::Packed;
        constexpr int N = sizeof(acc) / sizeof(acc[0]);
        const uint32_t ep = ++epoch;
        warp_scatter_sums<N, A>(acc, reinterpret_cast<Pk*>(red[threadIdx.x >> 5]));
        __syncthreads();
        const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
        uint2* const slots = ra.pl + (ph * 8 + w) * kMaxBlocks * 2;
        // block 0's totals, a copy for every eighth block (fewer polls per line)
        uint2* const sums = ra.pl + 16 * kMaxBlocks * 2 + ph * 8 * 64;
        if (w < N) {
            A y;
            if (l < (int)(blockDim.x >> 5)) y = A::unpack(reinterpret_cast<Pk*>(red[l])[w]);
#pragma unroll
            for (int o = kResThreads / 64; o > 0; o >>= 1) y.shfl_add(o);
            Pk mine = y.pack();
            if (ra.cluster) {
                uint2 bits;
                mine = lane0(mine);
                memcpy(&bits, &mine, 8);
                if (l < nb) put_remote(&part[ph][w][blockIdx.x][0], l, bits, ep);
                y = A();
                if (l < nb) {
                    bits = get_shared(&part[ph][w][l][0], ep, wait);
                    memcpy(&mine, &bits, 8);
                    y = A::unpack(mine);
                }
#pragma unroll
                for (int o = kClusterBlocks / 2; o > 0; o >>= 1) y.shfl_add(o);
            } else if (nb > 1) {
                if (l == 0) put(slots, blockIdx.x, mine, ep);
                if (blockIdx.x == 0) {
                    constexpr int B = kMaxBlocks / 32;
                    Pk v[B];
                    get_all<B, Pk>(
                        v, [&](int u) FEA_INLINE { return l + 32 * u < nb; },
                        [&](int u, Pk& x) FEA_INLINE { return try_get<Pk>(slots, l + 32 * u, x, ep); }, wait);
                    y = A();
#pragma unroll
                    for (int u = 0; u < B; u++)
                        if (l + 32 * u < nb) y.merge(A::unpack(v[u]));
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) y.shfl_add(o);
                    mine = lane0(y.pack());  // (lanes may differ in the last bit)
                    if (l < 8) put(sums + l * 64, w, mine, ep);
                }
            }
            if (l == 0 && (ra.cluster || blockIdx.x == 0)) reinterpret_cast<Pk*>(tot)[w] = y.pack();
        }
        if (!ra.cluster && blockIdx.x != 0 && threadIdx.x < N)
            reinterpret_cast<Pk*>(tot)[threadIdx.x] = get<Pk>(sums + (blockIdx.x & 7) * 64, threadIdx.x, ep, wait);
        ph ^= 1;
        return __syncthreads_or(*wait.dead) == 0;  // the same answer in every thread
    };
    auto x_epoch = [&]() FEA_INLINE { return ++epoch != 0 ? epoch : ++epoch; };  // (0 has a meaning, below)
    auto total = [&](int k) FEA_INLINE { return Acc<R>::unpack(reinterpret_cast<typename Acc<R>::Packed*>(tot)[k]); };

    const int kind = ra.kind;
    const bool gs = kind == EQ_GS_REF || kind == EQ_GS_CONSISTENT;
    const bool stiff = a.ngrp > 0;
    bool prev_ok = gs && a.xprev && run->prev_valid != 0;
    uint32_t xep[2] = {0, 0};  // epochs of the two x buffers; 0: x (xprev) is in global memory

    V cr[kP], cw[kP], cs[kP], cx[kP], cp[kP], hr[kP], hs[kP], hw[kP];

    // Operands of the full layout (A, M, K, Adv): the row's own value and its halo's.
    auto stage = [&](auto own, auto halo) FEA_INLINE {
        __syncthreads();  // earlier reads of the staging buffers are done
#pragma unroll
        for (int q = 0; q < kP; q++) {
            const int tile = tile_of(q);
            if (tile < 0) continue;
            V* u = ub_of(q);
            u[t] = rowq[q] >= 0 ? own(q, row_of(q)) : V{};
            const int32_t h0 = __ldg(a.halo_off + tile), hc = __ldg(a.halo_off + tile + 1) - h0;
            if (j < hc) u[kTileRows + j] = halo((int64_t)__ldg(a.halo_col + h0 + j));
        }
        __syncthreads();
    };
    auto full_rows = [&](int q, auto add) FEA_INLINE {  // add(entry, staged operand) in CSR order
        const int tile = tile_of(q);
        if (tile < 0) return;
        const V* u = ub_of(q);
        const int32_t sb = __ldg(a.slice_off + tile * 8 + w8), sw = (__ldg(a.slice_off + tile * 8 + w8 + 1) - sb) >> 5;
#pragma unroll 4
        for (int k = 0; k < sw; k++) {
            const int32_t e = sb + 32 * k + lane;
            add(e, u[__ldg(a.lcol + e)]);
        }
    };
    // The row's product with the resident operator, added to w.
    auto product = [&](int q, V w) FEA_INLINE {
        const V* u = ub_of(q);
        const int base = (q * ra.tpb + grp) * emx + (sref[q] >> 16) + lane, sw = sref[q] & 0xffff;
#pragma unroll 4
        for (int k = 0; k < sw; k++) {
            const V av = ent[base + 32 * k];
            const V g = u[lcs[base + 32 * k]];
#pragma unroll
            for (int f = 0; f < NF; f++) w.v[f] = fmar(av.v[f], g.v[f], w.v[f]);
        }
        return w;
    };

    int done = 0, halt = 0;
    long long iters = 0;
    for (int step = 0; step < ra.steps; step++) {
        // ---- right-hand side b and r = b - A x0 -----------------------------------
        const StepParams prm = *a.prm;
        const R dt = (R)prm.dt;
        const bool extrap = prev_ok && run->guess == 1;
        const int xb = step & 1;  // x buffer of this step's result; the other holds x_n
        auto state = [&](int64_t i, bool halo) FEA_INLINE {  // x_n of row i
            return halo && xep[xb ^ 1] ? get<V>(ra.xl[xb ^ 1], i, xep[xb ^ 1], wait) : ldv(a.x + i, true);
        };
        auto guess = [&](const V& xn, int64_t i, bool halo) FEA_INLINE {  // the solve's start there
            V g = xn;
            if (extrap) {
                const V xp = halo && xep[xb] ? get<V>(ra.xl[xb], i, xep[xb], wait) : ldv(a.xprev + i, true);
#pragma unroll
                for (int f = 0; f < NF; f++) g.v[f] = fmar((R)2, xn.v[f], -xp.v[f]);
            }
            return g;
        };
        Acc<R> ax[kP][NF], bs[kP][NF];
        // wave: the second operand (u, or Newmark's predictor), sent to the halos
        const bool wave = kind == EQ_WAVE_REF || kind == EQ_NEWMARK_INIT || kind == EQ_WAVE_NEWMARK;
        const uint32_t wep = wave ? ++epoch : 0;
        if (wave) {
#pragma unroll
            for (int q = 0; q < kP; q++) {
                if (rowq[q] < 0) continue;
                const int64_t row = row_of(q);
                V y{};
                y.v[0] = a.u[row];
                if (kind == EQ_WAVE_NEWMARK) {
                    const R vr = a.v[row], ar = a.x[row].v[0];
                    y.v[0] = y.v[0] + dt * vr + dt * dt * ((R)0.5 - (R)prm.beta) * ar;
                    a.ut[row] = y.v[0];
                    a.vt[row] = vr + dt * ((R)1 - (R)prm.gamma) * ar;
                }
                put(ra.yl, row, y, wep);
                cx[q] = y;
            }
        }
        stage([&](int, int64_t i) FEA_INLINE { return guess(state(i, false), i, false); },
              [&](int64_t i) FEA_INLINE { return guess(state(i, true), i, true); });
#pragma unroll
        for (int q = 0; q < kP; q++)
            full_rows(q, [&](int32_t e, const V& g) FEA_INLINE {
                const V av = ldfv(a.As + e);
#pragma unroll
                for (int f = 0; f < NF; f++) ax[q][f].add_prod(av.v[f], g.v[f]);
            });
        auto add_term = [&](const R* m, auto coef) FEA_INLINE {  // bs += coef(m) * staged
#pragma unroll
            for (int q = 0; q < kP; q++)
                full_rows(q, [&](int32_t e, const V& g) FEA_INLINE {
                    const R me = coef(__ldg(m + e));
#pragma unroll
                    for (int f = 0; f < NF; f++) bs[q][f].add_prod(me, g.v[f]);
                });
        };
        if (kind == EQ_HEAT || kind == EQ_ADV_EXPLICIT || kind == EQ_WAVE_REF || kind == EQ_GS_REF) {
            if (extrap)
                stage([&](int, int64_t i) FEA_INLINE { return state(i, false); },
                      [&](int64_t i) FEA_INLINE { return state(i, true); });
            add_term(a.Ms, [&](R m) FEA_INLINE { return div_rn(m, dt); });
        }
        if (kind == EQ_ADV_EXPLICIT) {
            const R sg = (R)prm.adv_sign;
            add_term(ra.Advs, [&](R m) FEA_INLINE { return sg * m; });
        }
        if (wave) {
            const R c2 = (R)prm.c2;
            stage([&](int q, int64_t) FEA_INLINE { return cx[q]; },
                  [&](int64_t i) FEA_INLINE { return get<V>(ra.yl, i, wep, wait); });
            add_term(ra.Ks, [&](R m) FEA_INLINE { return -c2 * m; });
        }
        if constexpr (NF == 2) {
            if (kind == EQ_GS_CONSISTENT) {
                const R Fr = (R)prm.F, Kr = (R)prm.k;
                auto react = [&](const V& x) FEA_INLINE {
                    const R u = x.v[0], v = x.v[1], uvv = u * (v * v);
                    V w;
                    w.v[0] = u / dt - uvv + Fr * ((R)1 - u);
                    w.v[1] = v / dt + uvv - (Fr + Kr) * v;
                    return w;
                };
                stage([&](int, int64_t i) FEA_INLINE { return react(state(i, false)); },
                      [&](int64_t i) FEA_INLINE { return react(state(i, true)); });
                add_term(a.Ms, [](R m) FEA_INLINE { return m; });
            }
        }
        uint32_t rep = ++epoch;  // r's epoch
        {
            unsigned int flags = 0;
            Acc<R> dots[NV + 1];  // the last counts flagged threads: every block learns of them
#pragma unroll
            for (int q = 0; q < kP; q++) {
                cr[q] = V{};
                if (rowq[q] < 0) continue;
                const int64_t row = row_of(q);
                const V xr = ldv(a.x + row, true);
                if constexpr (NF == 2) {
                    if (kind == EQ_GS_REF) {  // nodal reaction, CPUSolver.cpp:134,137
                        const R Fr = (R)prm.F, Kr = (R)prm.k;
                        const R u = xr.v[0], v = xr.v[1], uvv = u * (v * v);
                        bs[q][0].add(-uvv);
                        bs[q][0].add(Fr * ((R)1 - u));
                        bs[q][1].add(uvv);
                        bs[q][1].add(-(Fr + Kr) * v);
                    }
                }
                if (kind == EQ_GIVEN) {  // adjoint values may be large: only non-finite stops
                    const V g = ldv(a.rhs + row, true);
#pragma unroll
                    for (int f = 0; f < NF; f++) {
                        bs[q][f].add(g.v[f]);
                        if (!isfinite(xr.v[f])) flags |= FEA_STATUS_NONFINITE;
                    }
                } else if (wave) {
                    flags |= check_value(a.u[row]) | check_value(a.v[row]);
                } else {
#pragma unroll
                    for (int f = 0; f < NF; f++) flags |= check_value(xr.v[f]);
                }
                const V d = ldfv(a.dinv + row);
                V bv, rv;
#pragma unroll
                for (int f = 0; f < NF; f++) {
                    bv.v[f] = bs[q][f].rounded();
                    bs[q][f].sub(ax[q][f]);
                    rv.v[f] = bs[q][f].rounded();
                    dots[f].add_prod(bv.v[f], bv.v[f]);
                    dots[NF + f].add_prod(rv.v[f], rv.v[f]);
                    dots[2 * NF + f].add_prod(rv.v[f], d.v[f] * rv.v[f]);
                }
                a.b[row] = bv;
                cr[q] = rv;
                put(ra.rl[0], row, rv, rep);
            }
            if (flags & (FEA_STATUS_BLOWUP | FEA_STATUS_NONFINITE)) dots[NV].add((R)1);
            raise_flags(run, flags);
            if (!reduce(dots)) break;
        }
        if (threadIdx.x == 0) {
            const int stop = total(NV).value() > 0.0;
            st.stop = sstop = stop;
            st.iter = 0;
            st.max_iter = run->max_iter;
            st.pending = 0;
#pragma unroll
            for (int f = 0; f < NF; f++)
                start_solve<R>((volatile CgState*)&st, f, stop, run->tol, total(f), total(NF + f), total(2 * NF + f));
        }
        __syncthreads();
        if (sstop) {
            halt = 1;
            break;
        }
        // ---- x_n to the history, the start to x -------------------------------------
        const bool send_x = gs && step == 0;  // the next step wants x_(n-1) at its halos
        if (send_x) xep[1] = x_epoch();
#pragma unroll
        for (int q = 0; q < kP; q++) {
            cx[q] = cp[q] = V{};
            if (rowq[q] < 0) continue;
            const int64_t row = row_of(q);
            const V xr = ldv(a.x + row, true);
            cx[q] = guess(xr, row, false);
            if (gs && a.xprev) a.xprev[row] = xr;
            if (send_x) put(ra.xl[1], row, xr, xep[1]);
        }
        prev_ok = gs && a.xprev;
        // ---- solve; then one true-residual pass, and fields above the tolerance restart -----
        bool failed = false;
        for (int round = 0;; round++) {
            int was[NF], any = 0;
#pragma unroll
            for (int f = 0; f < NF; f++) any |= was[f] = st.active[f];
            if (round > 0 && !any) break;
            uint32_t hep = rep;  // the halos' r: as published, or in the stiff groups' basis
            if (any && stiff) {
                // the members' rows into the basis (k_stiff_in), the start aside
                hep = ++epoch;
                double corr[NF];
#pragma unroll
                for (int f = 0; f < NF; f++) corr[f] = 0;
#pragma unroll
                for (int q = 0; q < kP; q++) {
                    if (rowq[q] < 0) continue;
                    const int64_t row = row_of(q);
                    const int wr = __ldg(ra.where + row);
                    if (wr >= 0) {
                        const V d = ldfv(a.dinv + row), di = cd[q];
                        double s[NF];
#pragma unroll
                        for (int f = 0; f < NF; f++) s[f] = 0;
                        for (int i = 0; i < 4; i++) {
                            const int m = __ldg(a.grp_mem + (wr & ~3) + i);
                            if (m < 0) continue;
                            const V rm = get<V>(ra.rl[0], m, rep, wait);
#pragma unroll
                            for (int f = 0; f < NF; f++)
                                s[f] += a.grp_Q[16 * ((int64_t)(wr >> 2) * NF + f) + 4 * i + (wr & 3)] * (double)rm.v[f];
                        }
#pragma unroll
                        for (int f = 0; f < NF; f++) {
                            const R rn = (R)s[f], z = d.v[f] * cr[q].v[f], zn = di.v[f] * rn;
                            corr[f] += (double)rn * (double)zn - (double)cr[q].v[f] * (double)z;
                            cr[q].v[f] = rn;
                        }
                        a.q[row] = cx[q];
                        cx[q] = V{};
                    }
                    put(ra.rl[1], row, cr[q], hep);
                }
                Acc<double> acc[NF];
#pragma unroll
                for (int f = 0; f < NF; f++) acc[f].s = corr[f];
                if (!reduce(acc)) {
                    failed = true;
                    break;
                }
                if (threadIdx.x == 0)
#pragma unroll
                    for (int f = 0; f < NF; f++) {
                        if (!st.active[f]) continue;
                        st.thr[f] = stiff_threshold<R>(st.thr[f]);
                        if constexpr (sizeof(R) == 4) {
                            const double g = (double)st.ffrz[f][0] + (double)st.ffrz[f][1] + tot[f];
                            st.rz[f] = g;
                            ff_store(st.ffrz[f], ff_of(g));
                            ff_store(st.ffthr[f], ff_of(st.thr[f]));
                        } else {
                            st.rz[f] += tot[f];
                        }
                    }
            }
            if (any) {
                // w0 = A z (the diagonal term is r), delta0 = z.w0
                __syncthreads();
                uint2* const rsrc = stiff ? ra.rl[1] : ra.rl[0];
#pragma unroll
                for (int q = 0; q < kP; q++) {
                    hr[q] = hs[q] = cs[q] = cw[q] = V{};
                    V* u = ub_of(q);
                    V z;
#pragma unroll
                    for (int f = 0; f < NF; f++) z.v[f] = cd[q].v[f] * cr[q].v[f];
                    if (tile_of(q) >= 0) u[t] = z;
                    if (hcol[q] >= 0) {
                        hr[q] = get<V>(rsrc, hcol[q], hep, wait);
#pragma unroll
                        for (int f = 0; f < NF; f++) z.v[f] = hd[q].v[f] * hr[q].v[f];
                        u[kTileRows + j] = z;
                    }
                }
                __syncthreads();
                uint32_t wep2 = ++epoch;
                {
                    Acc<R> acc[NF];  // exact products, as in the ring kernels' set-up
#pragma unroll
                    for (int q = 0; q < kP; q++) {
                        if (rowq[q] < 0) continue;
                        cw[q] = product(q, cr[q]);
                        put(ra.wl[0], rowq[q], cw[q], wep2);
                        const V z = ub_of(q)[t];
#pragma unroll
                        for (int f = 0; f < NF; f++) acc[f].add_prod(z.v[f], cw[q].v[f]);
                    }
                    if (!reduce(acc)) {
                        failed = true;
                        break;
                    }
                }
                if (threadIdx.x == 0) {
                    Acc<R> out[NF];
                    int act[NF];
#pragma unroll
                    for (int f = 0; f < NF; f++) {
                        out[f] = total(f);
                        act[f] = st.active[f];
                    }
                    finish_spmv<R, NF>((volatile CgState*)&st, &sflags, act, out);
                    ctl.any = 0;
#pragma unroll
                    for (int f = 0; f < NF; f++) {
                        ctl.act[f] = st.active[f];
                        ctl.any |= st.active[f];
                        ctl.alpha[f] = sizeof(R) == 4 ? (R)st.falpha[f] : (R)st.alpha[f];
                        ctl.beta[f] = 0;
                    }
                }
                __syncthreads();
                const int sf = (int)(threadIdx.x % NF);  // warp 0: the field of a lane's scalars
                int it = st.iter, sact = ctl.act[sf];
                const int most = st.max_iter;
                int more = ctl.any;
                for (int k = 0; more; k++) {
                    // the halos' w, wanted after the rows' updates
                    get_all<kP, V>(
                        hw, [&](int q) FEA_INLINE { return hcol[q] >= 0; },
                        [&](int q, V& x) FEA_INLINE { return try_get<V>(ra.wl[k & 1], hcol[q], x, wep2); }, wait);
                    PhaseCtl<R, NF> c;
                    c.need_old = k > 0;
#pragma unroll
                    for (int f = 0; f < NF; f++) {
                        c.act[f] = ctl.act[f];
                        c.fresh[f] = k == 0;
                        c.beta[f] = ctl.beta[f];
                        c.alpha[f] = c.act[f] ? ctl.alpha[f] : (R)0;
                    }
                    R dots[NV];
#pragma unroll
                    for (int i = 0; i < NV; i++) dots[i] = 0;
#pragma unroll
                    for (int q = 0; q < kP; q++) {
                        if (rowq[q] < 0) continue;
                        V sn, rn, un;
                        cg_advance(c, cr[q], cw[q], k > 0 ? cs[q] : cw[q], cd[q], sn, rn, un);
#pragma unroll
                        for (int f = 0; f < NF; f++) {
                            if (c.act[f]) {
                                const R ui = cd[q].v[f] * cr[q].v[f];
                                cp[q].v[f] = c.fresh[f] ? ui : fmar(c.beta[f], cp[q].v[f], ui);
                                cx[q].v[f] = fmar(c.alpha[f], cp[q].v[f], cx[q].v[f]);
                            }
                            dots[f] = fmar(rn.v[f], un.v[f], dots[f]);
                            dots[2 * NF + f] = fmar(rn.v[f], rn.v[f], dots[2 * NF + f]);
                        }
                        cr[q] = rn;
                        cs[q] = sn;
                        ub_of(q)[t] = un;
                    }
#pragma unroll
                    for (int q = 0; q < kP; q++) {
                        if (hcol[q] < 0) continue;
                        V sn, rn, un;
                        cg_advance(c, hr[q], hw[q], k > 0 ? hs[q] : hw[q], hd[q], sn, rn, un);
                        hr[q] = rn;
                        hs[q] = sn;
                        ub_of(q)[kTileRows + j] = un;
                    }
                    __syncthreads();
                    wep2 = ++epoch;
#pragma unroll
                    for (int q = 0; q < kP; q++) {
                        if (rowq[q] < 0) continue;
                        cw[q] = product(q, cr[q]);
                        put(ra.wl[(k & 1) ^ 1], opaque(rowq[q]), cw[q], wep2);
                        const V un = ub_of(q)[t];
#pragma unroll
                        for (int f = 0; f < NF; f++) dots[NF + f] = fmar(cw[q].v[f], un.v[f], dots[NF + f]);
                    }
                    Acc<R> acc[NV];
#pragma unroll
                    for (int i = 0; i < NV; i++) acc[i].add(dots[i]);
                    if (!reduce(acc)) {
                        failed = true;
                        break;
                    }
                    // The CG scalars as finish_cgcg computes them, in warp 0: beta = g / gamma,
                    // den = delta - beta (g / alpha), alpha = g / den.  The first two divisions
                    // run side by side, lanes below NF taking g / gamma and the next NF
                    // g / alpha.  They are divisions: a product with a kept reciprocal rounds
                    // once more and overflows where gamma is below 2^-128.
                    if (threadIdx.x < 32) {
                        const Acc<R> ag = total(sf), ad = total(NF + sf), rr = total(2 * NF + sf);
                        it++;
                        int state = 0;  // 0: iterates, 1: converged, 2: breakdown
                        R al = 0, be = 0;
                        volatile CgState* const sv = &st;  // gamma and alpha live there: fewer registers
                        const bool second = threadIdx.x >= NF;
                        if constexpr (sizeof(R) == 4) {
                            const FF r2 = ff_norm(rr), g = ff_norm(ag);
                            const FF quot = ff_div(g, ff_load(second ? sv->ffalpha[sf] : sv->ffrz[sf]));
                            const FF beta = from_lane(quot, sf), ga = from_lane(quot, NF + sf);
                            const FF den = ff_sub(ff_norm(ad), ff_mul(beta, ga));
                            const FF alpha = ff_div(g, den);
                            al = alpha.rounded();
                            be = beta.rounded();
                            state = !isfinite(r2.hi) ? 2
                                    : ff_less(r2, ff_load(sv->ffthr[sf])) ? 1
                                    : !(den.hi > 0.f) || !isfinite(alpha.hi) || !isfinite(beta.hi) ? 2
                                                                                                    : 0;
                            if (threadIdx.x < NF) {
                                ff_store(sv->ffrz[sf], g);
                                ff_store(sv->ffalpha[sf], alpha);
                            }
                        } else {
                            const double g = ag.s, quot = g / (second ? sv->alpha[sf] : sv->rz[sf]);
                            const double beta = __shfl_sync(0xffffffffu, quot, sf),
                                         ga = __shfl_sync(0xffffffffu, quot, NF + sf);
                            const double den = ad.s - beta * ga, alpha = g / den;
                            al = alpha;
                            be = beta;
                            state = !isfinite(rr.s) ? 2
                                    : rr.s < sv->thr[sf] ? 1
                                    : !(den > 0.0) || !isfinite(alpha) || !isfinite(beta) ? 2
                                                                                          : 0;
                            if (threadIdx.x < NF) {
                                sv->rz[sf] = g;
                                sv->alpha[sf] = alpha;
                            }
                        }
                        const bool on = sact && state == 0;
                        const bool cont = __any_sync(0xffffffffu, on) && it < most;
                        if (threadIdx.x < NF) {
                            ctl.alpha[sf] = al;
                            ctl.beta[sf] = be;
                            ctl.act[sf] = on && cont;
                            if (sact && !(on && cont)) {
                                st.active[sf] = 0;
                                st.iters[sf] = it;
                                st.rr[sf] = rr.value();
                                // (the limit is judged by the caller's tolerance, not the groups' stricter stop)
                                if (state == 2) atomicOr(&sflags, FEA_STATUS_BREAKDOWN);
                                else if (state == 0 && !(stiff && rr.value() < run->tol * run->tol * st.bb[sf]))
                                    atomicOr(&sflags, FEA_STATUS_NOT_CONVERGED);
                            }
                        }
                        if (threadIdx.x == 0) ctl.any = cont;
                        sact = on && cont;
                    }
                    __syncthreads();
                    more = ctl.any;
                }
                if (failed) break;
                if (threadIdx.x == 0) st.iter = it;
                if (stiff) {
                    // x = x0 + Q y on the members' rows (k_stiff_out)
                    const uint32_t yep = ++epoch;
#pragma unroll
                    for (int q = 0; q < kP; q++) {
                        if (rowq[q] < 0) continue;
                        const int64_t row = row_of(q);
                        if (__ldg(ra.where + row) >= 0) put(ra.rl[1], row, cx[q], yep);
                    }
#pragma unroll
                    for (int q = 0; q < kP; q++) {
                        if (rowq[q] < 0) continue;
                        const int64_t row = row_of(q);
                        const int wr = __ldg(ra.where + row);
                        if (wr < 0) continue;
                        V x = a.q[row];
                        double s[NF];
#pragma unroll
                        for (int f = 0; f < NF; f++) s[f] = x.v[f];
                        for (int i = 0; i < 4; i++) {
                            const int m = __ldg(a.grp_mem + (wr & ~3) + i);
                            if (m < 0) continue;
                            const V y = get<V>(ra.rl[1], m, yep, wait);
#pragma unroll
                            for (int f = 0; f < NF; f++)
                                s[f] += a.grp_Q[16 * ((int64_t)(wr >> 2) * NF + f) + 4 * (wr & 3) + i] * (double)y.v[f];
                        }
#pragma unroll
                        for (int f = 0; f < NF; f++) cx[q].v[f] = (R)s[f];
                    }
                    if (threadIdx.x == 0)
#pragma unroll
                        for (int f = 0; f < NF; f++)
                            if (was[f]) st.thr[f] = solve_threshold<R>(run->tol, st.bb[f]);
                }
                if (__syncthreads_or(*wait.dead)) {  // (the members' values came after the last reduction)
                    failed = true;
                    break;
                }
            }
            // x to global memory and to the halos; zero right-hand sides give x = 0
            xep[xb] = x_epoch();
#pragma unroll
            for (int q = 0; q < kP; q++) {
                if (rowq[q] < 0) continue;
                const int64_t row = row_of(q);
#pragma unroll
                for (int f = 0; f < NF; f++)
                    if (!(st.bb[f] > 0.0)) cx[q].v[f] = 0;
                a.x[row] = cx[q];
                put(ra.xl[xb], row, cx[q], xep[xb]);
            }
            const int mode = run->refine;
            if (round > 0 || !mode || st.iter >= st.max_iter) break;
            rep = ++epoch;
            stage([&](int q, int64_t) FEA_INLINE { return cx[q]; },
                  [&](int64_t i) FEA_INLINE { return get<V>(ra.xl[xb], i, xep[xb], wait); });
            auto residual = [&](auto tag) FEA_INLINE -> bool {
                using A = decltype(tag);
                A dots[2 * NF];
#pragma unroll
                for (int q = 0; q < kP; q++) {
                    A sum[NF];
                    full_rows(q, [&](int32_t e, const V& g) FEA_INLINE {
                        const V av = ldfv(a.As + e);
#pragma unroll
                        for (int f = 0; f < NF; f++) sum[f].add_prod(av.v[f], g.v[f]);
                    });
                    if (rowq[q] < 0) continue;
                    const int64_t row = row_of(q);
                    const V bv = a.b[row], d = ldfv(a.dinv + row);
#pragma unroll
                    for (int f = 0; f < NF; f++) {
                        A s;
                        s.add(bv.v[f]);
                        s.sub(sum[f]);
                        cr[q].v[f] = (R)s.rounded();
                        dots[f].add_prod(cr[q].v[f], cr[q].v[f]);
                        dots[NF + f].add_prod(cr[q].v[f], d.v[f] * cr[q].v[f]);
                    }
                    put(ra.rl[0], row, cr[q], rep);
                }
                if (!reduce(dots)) return false;
                if (threadIdx.x == 0)
#pragma unroll
                    for (int f = 0; f < NF; f++) {
                        const A rr = A::unpack(reinterpret_cast<typename A::Packed*>(tot)[f]),
                                rz = A::unpack(reinterpret_cast<typename A::Packed*>(tot)[NF + f]);
                        st.active[f] = 0;
                        st.fresh[f] = 1;
                        if (!(st.bb[f] > 0.0)) continue;
                        st.rr[f] = rr.value();
                        if (rr.value() < st.thr[f]) continue;
                        if constexpr (std::is_same_v<A, Acc<R>>) {
                            set_gamma((volatile CgState*)&st, f, rz);
                        } else {  // FP64 norms of an FP32 handle
                            st.rz[f] = rz.value();
                            ff_store(st.ffrz[f], ff_of(rz.value()));
                        }
                        st.active[f] = 1;
                    }
                __syncthreads();
                return true;
            };
            bool ok;
            if constexpr (sizeof(R) == 4) ok = mode == 2 ? residual(Acc<double>{}) : residual(Acc<R>{});
            else ok = residual(Acc<R>{});
            if (!ok) {
                failed = true;
                break;
            }
        }
        if (failed) break;
        // ---- wave updates (k_post), bookkeeping ---------------------------------------
        if (kind == EQ_WAVE_REF || kind == EQ_WAVE_NEWMARK) {
#pragma unroll
            for (int q = 0; q < kP; q++) {
                if (rowq[q] < 0) continue;
                const int64_t row = row_of(q);
                const R x = cx[q].v[0];
                if (kind == EQ_WAVE_REF) {
                    a.u[row] = a.u[row] + x * dt;
                } else {
                    a.u[row] = a.ut[row] + (R)prm.beta * dt * dt * x;
                    a.v[row] = a.vt[row] + (R)prm.gamma * dt * x;
                }
            }
        }
        done++;
        iters += st.iter;
        if (threadIdx.x == 0)  // the next step's start rewrites them, and it may stop there
#pragma unroll
            for (int f = 0; f < NF; f++) {
                last.iters[f] = st.iters[f];
                last.rr[f] = st.rr[f];
                last.bb[f] = st.bb[f];
            }
    }
    if (ra.cluster) cluster_barrier();  // no block leaves while another may write into it
    // a wait expired here: whichever block it was, the call's later launches do
    // nothing and its step count leaves out the steps this block did not finish
    if (dead && threadIdx.x == 0) {
        atomicOr(&run->flags, FEA_STATUS_BREAKDOWN);
        atomicExch(&run->halt, 1);
        atomicExch(&run->expired, 1);
        atomicMax(&run->lost, ra.left - done);
    }
    // has_numerical_instability of the final state (k_final_check)
    unsigned int flags = 0;
#pragma unroll
    for (int q = 0; q < kP; q++) {
        if (rowq[q] < 0) continue;
        const int64_t row = row_of(q);
        if (kind == EQ_WAVE_REF || kind == EQ_WAVE_NEWMARK || kind == EQ_NEWMARK_INIT) {
            flags |= check_value(a.u[row]) | check_value(a.v[row]);
        } else {
            const V x = ldv(a.x + row, true);
#pragma unroll
            for (int f = 0; f < NF; f++)
                flags |= kind == EQ_GIVEN ? (isfinite(x.v[f]) ? 0u : FEA_STATUS_NONFINITE) : check_value(x.v[f]);
        }
    }
    raise_flags(run, flags);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (sflags) atomicOr(&run->flags, sflags);
        if (halt) atomicExch(&run->halt, 1);
        run->epoch = epoch + (dead ? 1u << 20 : 0u);  // past anything another block may have sent
        run->steps_done = (ra.first ? 0 : run->steps_done) + done;
        run->steps_left = 0;
        run->total_iters += iters;
        run->cg_launches += iters;
        if (done > 0) {
            for (int f = 0; f < NF; f++) {
                run->last_iters[f] = last.iters[f];
                run->last_rel[f] = last.bb[f] > 0.0 ? sqrt(last.rr[f] / last.bb[f]) : 0.0;
            }
            if (gs && a.xprev) run->prev_valid = 1;
        }
    }
}

template <typename R, int NF>
using ResidentFn = void (*)(StepArgs<R, NF>, ResidentArgs<R>);

// The kernel for `passes` tiles per thread group, or null: up to where the step
// graph is faster.  A pass keeps 9 to 36 registers by type and fields, and every
// instance uses all 128 of a thread and spills the rest
// (bytes of spill stores for one pass and for the most:
// FP32 one field 204 and 396, two fields 244 and 1004, FP64 one field 0 and 432, two
// fields 92 and 408).  At 17 tiles a block (the level-8 icosphere, one FP32
// field) nine passes ran 50 Newmark steps in 16.5 ms, the step graph in 10.0.
template <typename R, int NF>
ResidentFn<R, NF> resident_kernel(int passes) {
    if (passes <= 1) return k_resident<R, NF, 1>;
    if (passes <= 2) return k_resident<R, NF, 2>;
    if constexpr (sizeof(R) * NF <= 8) {
        if (passes <= 3) return k_resident<R, NF, 3>;
        if (passes <= 4) return k_resident<R, NF, 4>;
    }
    // (a sixth pass spills too much: heat, 640 x 640 grid, 48.2 ms against the
    // graph's 39.2; five passes, 590 x 590, 28.5 against 33.0)
    if constexpr (sizeof(R) * NF == 4)
        if (passes <= 5) return k_resident<R, NF, 5>;
    return nullptr;
}

// One cluster, or a cooperative grid.
cudaLaunchConfig_t launch_config(const ResidentPlan& p, cudaLaunchAttribute& attr, cudaStream_t st) {
    attr = cudaLaunchAttribute{};
    if (p.cluster) {
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = (unsigned)p.blocks;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    } else {
        attr.id = cudaLaunchAttributeCooperative;
        attr.val.cooperative = 1;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)p.blocks);
    cfg.blockDim = dim3((unsigned)(p.tpb * kTileRows));
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = p.blocks > 1 ? 1 : 0;
    return cfg;
}

}  // namespace

template <typename R, int NF>
bool plan_resident(const StepArgs<R, NF>& a, ResidentPlan& p) {
    p = ResidentPlan{};
    if (!a.As || !a.As_od || !a.Ms || a.N <= 0) return false;
    const int us = kTileRows + std::max(a.hmax, a.hmax_od);
    // one halo slot per row thread; slices named by 15-bit offsets
    if (us > 2 * kTileRows || a.emax_od > 32767) return false;
    const int64_t ntiles = ceil_div(a.N, kTileRows);
    const int64_t most = std::min(num_sms(), kMaxBlocks);
    // up to two tiles in one block (no exchange at all), then one cluster, then
    // the whole device, as few tiles a block as it has SMs for (two a block on
    // half the blocks: heat, 142 tiles, 3,351 against 3,135 us, Gray-Scott 2,673
    // against 2,449)
    p.cluster = ntiles > 2 && ntiles <= kClusterBlocks * kClusterTiles<R>;
    int64_t T = ntiles <= 2 ? ntiles : ceil_div(ntiles, p.cluster ? (int64_t)kClusterBlocks : most);
    const auto al = [](size_t x) { return (x + 15) & ~(size_t)15; };
    p.T = (int)T;
    p.blocks = (int)ceil_div(ntiles, T);
    p.passes = (int)ceil_div(T, kResThreads / kTileRows);
    p.tpb = (int)ceil_div(T, p.passes);
    p.smem = al((size_t)T * a.emax_od * sizeof(FV<R, NF>)) + al((size_t)T * a.emax_od * 2) +
             (size_t)T * us * sizeof(FV<R, NF>);
    p.us = us;
    const ResidentFn<R, NF> fn = resident_kernel<R, NF>(p.passes);
    if (p.smem > (size_t)200 * 1024 || !fn) return false;
    ensure_dyn_smem(fn, p.smem);
    int n = 0;
    if (p.cluster) {
        int c = 1;
        while (c < p.blocks) c *= 2;  // blocks without tiles only take part in the reductions
        p.blocks = c;
        cudaLaunchAttribute attr;
        const cudaLaunchConfig_t cfg = launch_config(p, attr, nullptr);
        if ((c > 8 && cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) ||
            cudaOccupancyMaxActiveClusters(&n, fn, &cfg) != cudaSuccess) {
            (void)cudaGetLastError();
            return false;
        }
        return n >= 1;
    }
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, p.tpb * kTileRows, p.smem) != cudaSuccess) {
        (void)cudaGetLastError();
        return false;
    }
    return (int64_t)n * num_sms() >= p.blocks;
}

template <typename R, int NF>
size_t resident_exchange_bytes(int64_t N) {
    const size_t rows = (size_t)(ceil_div(N, kTileRows) * kTileRows);
    return rows * sizeof(FV<R, NF>) * 2 * 7 + sizeof(uint2) * (2 * 16 * kMaxBlocks + 2 * 8 * 64);
}

template <typename R, int NF>
void run_resident(const StepArgs<R, NF>& a, const ResidentPlan& p, const R* Ks, const R* Advs, const int32_t* where,
                  void* exchange, int kind, int64_t nsteps, cudaStream_t st) {
    const ResidentFn<R, NF> fn = resident_kernel<R, NF>(p.passes);  // opted in to p.smem by plan_resident
    ResidentArgs<R> ra{};
    ra.kind = kind;
    ra.T = p.T;
    ra.tpb = p.tpb;
    ra.us = p.us;
    ra.Ks = Ks;
    ra.Advs = Advs;
    ra.where = where;
    uint2* at = (uint2*)exchange;
    const int64_t pairs = ceil_div(a.N, kTileRows) * kTileRows * kPairs<FV<R, NF>>;
    for (uint2** buf : {&ra.wl[0], &ra.wl[1], &ra.xl[0], &ra.xl[1], &ra.rl[0], &ra.rl[1], &ra.yl}) {
        *buf = at;
        at += pairs;
    }
    ra.pl = at;
    ra.cluster = p.cluster;
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = launch_config(p, attr, st);
    ra.wait = kWaitClocks;
    if (const char* most = getenv("FEA_WAIT_CLOCKS"))
        if (const long long n = strtoll(most, nullptr, 10); n > 0) ra.wait = n;
    for (int64_t s0 = 0; s0 < nsteps; s0 += kResidentSteps) {
        ra.left = nsteps - s0;
        ra.first = s0 == 0;
        ra.steps = (int)std::min<int64_t>(kResidentSteps, nsteps - s0);
        FEA_CUDA_TRY(cudaLaunchKernelEx(&cfg, fn, a, ra));
    }
}

#define FEA_INST_RES(R, NF)                                                                                     \
    template bool plan_resident<R, NF>(const StepArgs<R, NF>&, ResidentPlan&);                                  \
    template size_t resident_exchange_bytes<R, NF>(int64_t);                                                    \
    template void run_resident<R, NF>(const StepArgs<R, NF>&, const ResidentPlan&, const R*, const R*,          \
                                      const int32_t*, void*, int, int64_t, cudaStream_t);
FEA_INST_RES(float, 1)
FEA_INST_RES(float, 2)
FEA_INST_RES(double, 1)
FEA_INST_RES(double, 2)

}  // namespace fea
