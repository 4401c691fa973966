// Resident iterations: an LP (or QP) whose matrices fit the GPU's shared memory
// iterates in one cooperative launch.
//
// A pass over a matrix of up to a million nonzeros is latency, not bandwidth:
// launch, row offsets -> column index -> gathered value through L2, epilogue,
// next launch. Here every CTA (one per SM) keeps its contiguous range of rows
// of A and of columns (rows of A') in shared memory for the whole launch --
// values, indices, bounds, iterates -- and only the two gathered vectors go
// through L2: a pass gathers, multiplies, sums its rows and writes its own
// slice of the other vector, and one grid barrier orders the passes. The
// gathers are taken nonzero by nonzero (every thread the same number in
// flight, whatever the row lengths) and in column order (RsPacked), the products
// staged in shared memory in row order and the row sums taken from there.
//
// The grid barrier spins on a counter in L2 (2,550 cycles with 148 CTAs;
// flags polled by every CTA and a two-level tree took 4,300-7,300, and packets
// of value and iteration number, which need no barrier, no less than it once
// their lines are shared by many readers). The launch is cooperative, so all
// CTAs are resident; the spin is bounded, and a CTA that gives up records the
// timeout in the device error flag and leaves, as the others then do.
#pragma once

#include "vk_csr.cuh"

#include <type_traits>

namespace vk {

constexpr int kRsThreads = 768;     // threads of a CTA, at most
constexpr int kRsSmem = 220 * 1024; // dynamic shared memory of a CTA (227 KB less the static part)
constexpr int kRsRowCost = 4;       // partition: a row costs this many nonzeros
// gathers in flight per thread: 50,000 x 100,000 LP 9.5 us an iteration with 2 or 4, 10.4 with 6
// or 8; QP 40,000 x 100,000 13.2 / 13.6 / 14.8 / 15.5; 4,000 x 8,000 6.4 / 6.1 / 6.5 / 7.0
constexpr int kRsGather = 4;
constexpr int kRsWarpRow = 32;      // a row of more than this many products per lane goes to a whole warp
constexpr int kRsMaxGrid = 160;
// Iterations in one launch, about: a launch holds the shared memory of every SM, and
// other streams' kernels that need some wait for its end. A 2,048 x 2,048 bf16 product
// beside solves of a 2,000 x 5,000 / 50,000 x 100,000 LP: 0.04-1.2 / 2.2 ms, with 1,024
// iterations a launch 4.7 / 9.2 ms (alone 0.035); the solves themselves take 0.2-0.7%
// longer (3.66 -> 3.69, 6.78 -> 6.81, 6.79 -> 6.81 ms).
constexpr int kRsLaunch = 256;
constexpr int kRsLook = 1024; // iterations between two looks of the host, about
constexpr unsigned kRsPolls = 1u << 25; // over ten seconds

// ---- device side ----------------------------------------------------------------

// One CTA's share of a matrix, in shared memory.
template <class T, class I>
struct RsSide {
    const T *v;
    const I *idx;
    const int *ro;
    int rows, nnz, L;
    bool longs; // some row goes to a whole warp
};

// The index of a nonzero that is gathered in column order: its column, and its
// place in the share (row order), where its product goes. A warp's gathers then
// share cache lines, and an L1 looks up one line a cycle (a share of 4,000
// nonzeros has 4,000 lookups in row order and 2,300-3,000 lines); the products
// land in the same places, so that the sums stay what they were. Measured, per
// float64 Halpern iteration: 4,000 x 8,000 LP with 240,000 nonzeros 9.02 -> 6.13 us,
// 50,000 x 100,000 with 600,000 10.44 -> 9.52, QP 40,000 x 100,000 15.75 -> 13.71, a
// power law of 528,000 12.01 -> 9.80, 2,000 x 5,000 with 40,000 5.14 -> 5.12 (float32,
// with the float64 finish: 10.57 -> 6.31, 11.06 -> 8.85, 13.00 -> 10.71, 13.26 -> 9.40).
// Hence every plan whose columns and shares its bits can hold is packed, unless
// only 16-bit indices leave room for the matrices.
struct RsPacked {
    static constexpr int kPlaceBits = 13, kColBits = 32 - kPlaceBits;
    uint32_t w;
};
template <class I>
__device__ __forceinline__ int rs_col(I i) { return static_cast<int>(i); }
__device__ __forceinline__ int rs_col(RsPacked i) { return static_cast<int>(i.w >> RsPacked::kPlaceBits); }
template <class I>
__device__ __forceinline__ int rs_place(I, int k) { return k; }
__device__ __forceinline__ int rs_place(RsPacked i, int) {
    return static_cast<int>(i.w & ((1u << RsPacked::kPlaceBits) - 1u));
}

template <class T, class I>
__device__ RsSide<T, I> rs_load(const int *__restrict__ ro, const int *__restrict__ ci, const T *__restrict__ val,
                                int r0, int r1, T *v, I *idx, int *sro) {
    const int k0 = ro[r0], nnz = ro[r1] - k0, rows = r1 - r0;
    for (int k = threadIdx.x; k < nnz; k += blockDim.x) {
        const int w = __ldg(ci + k0 + k);
        if constexpr (std::is_same_v<I, RsPacked>) { // ci: the plan's packed words
            idx[k] = RsPacked{static_cast<uint32_t>(w)};
            v[k] = __ldg(val + k0 + rs_place(idx[k], k));
        } else {
            idx[k] = static_cast<I>(w);
            v[k] = __ldg(val + k0 + k);
        }
    }
    // lanes per row: every thread busy in one round, at most about one per nonzero
    int L = 1;
    while (L < 32 && rows * L * 2 <= static_cast<int>(blockDim.x) && rows * L < nnz) L *= 2;
    bool lone = false;
    for (int r = threadIdx.x; r <= rows; r += blockDim.x) {
        sro[r] = ro[r0 + r] - k0;
        lone = lone || (r < rows && ro[r0 + r + 1] - ro[r0 + r] > kRsWarpRow * L);
    }
    return RsSide<T, I>{v, idx, sro, rows, nnz, L, __syncthreads_or(lone) != 0};
}

// prod[k] = v_k x[idx_k]; x is written by other CTAs during the launch. A:
// the products' type (float64 in the checks).
template <class A, class T, class I>
__device__ __forceinline__ void rs_products(const RsSide<T, I> &s, const T *x, A *prod) {
    const int nt = blockDim.x;
    int k = threadIdx.x;
    for (; k + (kRsGather - 1) * nt < s.nnz; k += kRsGather * nt) {
        T g[kRsGather];
        I i[kRsGather];
#pragma unroll
        for (int u = 0; u < kRsGather; ++u) {
            i[u] = s.idx[k + u * nt];
            g[u] = __ldcg(x + rs_col(i[u]));
        }
#pragma unroll
        for (int u = 0; u < kRsGather; ++u)
            prod[rs_place(i[u], k + u * nt)] = static_cast<A>(s.v[k + u * nt]) * static_cast<A>(g[u]);
    }
    if (k < s.nnz) { // fewer than kRsGather left
        T g[kRsGather];
        I i[kRsGather];
#pragma unroll
        for (int u = 0; u < kRsGather; ++u)
            if (k + u * nt < s.nnz) {
                i[u] = s.idx[k + u * nt];
                g[u] = __ldcg(x + rs_col(i[u]));
            }
#pragma unroll
        for (int u = 0; u < kRsGather; ++u)
            if (k + u * nt < s.nnz)
                prod[rs_place(i[u], k + u * nt)] = static_cast<A>(s.v[k + u * nt]) * static_cast<A>(g[u]);
    }
}

// The sum over a group of L lanes, in every one of them.
template <class A>
__device__ __forceinline__ A rs_group_sum(A v, int L) {
    const unsigned FULL = 0xffffffffu;
    if (L > 16) v += __shfl_xor_sync(FULL, v, 16);
    if (L > 8) v += __shfl_xor_sync(FULL, v, 8);
    if (L > 4) v += __shfl_xor_sync(FULL, v, 4);
    if (L > 2) v += __shfl_xor_sync(FULL, v, 2);
    if (L > 1) v += __shfl_xor_sync(FULL, v, 1);
    return v;
}

// Waits for the block's products, then row(r, sum, pre(r)) for every row, in
// one lane of the row's group; the first rows' bounds and pre(r) are fetched
// before the wait (2,000 x 5,000 LP 5.36 -> 5.17 us an iteration, 50,000 x
// 100,000 10.63 -> 10.31).
template <class A, class T, class I, class P, class F>
__device__ __forceinline__ void rs_rows(const RsSide<T, I> &s, const A *prod, P &&pre, F &&row) {
    const unsigned FULL = 0xffffffffu;
    const int L = s.L, lane = threadIdx.x & 31, sl = lane & (L - 1);
    const int step = static_cast<int>(blockDim.x) / L;
    int r = static_cast<int>(threadIdx.x) / L;
    int rb = (static_cast<int>(threadIdx.x) & ~31) / L; // the warp's first row: uniform trip count
    bool valid = r < s.rows;
    int a = valid ? s.ro[r] : 0, b = valid ? s.ro[r + 1] : 0;
    decltype(pre(0)) in{};
    if (valid) in = pre(r);
    __syncthreads();
    while (rb < s.rows) {
        A acc = A(0);
        const bool lone = s.longs && b - a > kRsWarpRow * L; // summed by the whole warp below
        if (!lone)
            for (int k = a + sl; k < b; k += L) acc += prod[k];
        acc = rs_group_sum(acc, L);
        if (s.longs) {
            unsigned lm = __ballot_sync(FULL, lone && sl == 0);
            while (lm) {
                const int src = __ffs(lm) - 1;
                const int fa = __shfl_sync(FULL, a, src), fb = __shfl_sync(FULL, b, src);
                A part = A(0);
                for (int k = fa + lane; k < fb; k += 32) part += prod[k];
                part = warp_sum(part);
                if (lane == src) acc = part;
                lm &= lm - 1u;
            }
        }
        if (valid && sl == 0) row(r, acc, in);
        rb += step;
        r += step;
        if (rb >= s.rows) break;
        valid = r < s.rows;
        a = valid ? s.ro[r] : 0;
        b = valid ? s.ro[r + 1] : 0;
        if (valid) in = pre(r);
    }
}
// The same for rows without inputs.
template <class A, class T, class I, class F>
__device__ __forceinline__ void rs_rows(const RsSide<T, I> &s, const A *prod, F &&row) {
    rs_rows(s, prod, [](int) { return 0; }, [&](int r, A sum, int) { row(r, sum); });
}

// A CTA's block barrier at the end of a grid barrier: false when the thread that
// waited gave up (`ok` false), after recording that.
__device__ __forceinline__ bool rs_block(bool ok, int *err) {
    if (!ok) atomicCAS(err, 0, static_cast<int>(kDevErrGridTimeout));
    return __syncthreads_or(!ok) == 0;
}

// The warp's maximum of v >= 0 (no NaN): such doubles order as their bits do, so
// that two integer reductions do for five steps of shuffles and comparisons.
__device__ __forceinline__ double rs_warp_max(double v) {
    const unsigned hi = static_cast<unsigned>(__double2hiint(v)), lo = static_cast<unsigned>(__double2loint(v));
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
    return __hiloint2double(static_cast<int>(mh), static_cast<int>(ml));
}

// Grid barrier over the gridDim.x CTAs of a cooperative launch; `counter` is
// zero at the launch. All writes before it are visible after it.
struct RsBarrier {
    unsigned *counter;
    int *err;
    unsigned target = 0;

    // False when another CTA never came: the caller returns.
    __device__ __forceinline__ bool sync() {
        __syncthreads();
        return arrive_and_wait();
    }
    // The same, and *slot becomes the largest of itself and every thread's v
    // (non-negative; NaN ignored). `warps`: 32 doubles of shared memory.
    __device__ __forceinline__ bool sync_max(double v, double *warps, double *slot) {
        v = rs_warp_max(v);
        if ((threadIdx.x & 31) == 0) warps[threadIdx.x >> 5] = v;
        __syncthreads();
        if (threadIdx.x < 32) {
            v = rs_warp_max(threadIdx.x < blockDim.x / 32 ? warps[threadIdx.x] : 0.0);
            if (threadIdx.x == 0) atomic_max_nonneg(slot, v);
        }
        return arrive_and_wait();
    }

private:
    __device__ __forceinline__ bool arrive_and_wait() {
        target += gridDim.x;
        bool ok = true;
        if (threadIdx.x == 0) {
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
            unsigned now = 0, polls = 0;
            do {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(now) : "l"(counter) : "memory");
            } while (static_cast<int>(now - target) < 0 && ++polls < kRsPolls);
            ok = static_cast<int>(now - target) >= 0;
        }
        return rs_block(ok, err);
    }
};

// Sums v over the grid in CTA order: out[r] (shared memory) holds the totals
// after it, in every CTA. `partials`: kRsMaxGrid * NR doubles in global memory.
template <int NR>
__device__ __forceinline__ bool rs_sum(double (&v)[NR], double *partials, double *scratch, double *out, RsBarrier &bar) {
    block_sum<NR>(v, scratch);
    if (threadIdx.x == 0)
        for (int r = 0; r < NR; ++r) partials[static_cast<size_t>(blockIdx.x) * NR + r] = v[r];
    if (!bar.sync()) return false;
    const int lane = threadIdx.x & 31;
    for (int r = static_cast<int>(threadIdx.x) >> 5; r < NR; r += static_cast<int>(blockDim.x) / 32) {
        double t = 0.0;
        for (int b = lane; b < static_cast<int>(gridDim.x); b += 32) t += __ldcg(partials + static_cast<size_t>(b) * NR + r);
        t = warp_sum(t);
        if (lane == 0) out[r] = t;
    }
    __syncthreads();
    return true;
}

// ---- host side (vk_resident.cu) ------------------------------------------------------

// The launch of a model: its shape, the largest shares, the shares' boundaries.
struct RsPlan {
    bool small = false;  // 16-bit indices
    bool packed = false; // gathers in column order (RsPacked): the bits can hold them
    int grid = 0, threads = 0;
    int cap_a = 0, cap_t = 0, cap_q = 0, rows = 0, cols = 0;
    DevBuf<int> part_a, part_t;
    DevBuf<unsigned> counter; // of the grid barrier
    DevBuf<int> words_a, words_t, words_q; // rs_pack: RsPacked, share by share
    // the index array of a launch
    const int *index(const DevBuf<int> &words, const CsrPattern32 &p, bool use_packed) const {
        return use_packed ? words.get() : p.ci.get();
    }
};

// Fills `plan` for A, its transpose and (or null) Q, without the packed words;
// false when the matrices can not fit in any precision, or a kernel variant is
// pinned. `ctas`: that many shares (0: rs_grid's).
bool rs_plan(const CsrPattern32 &a, const CsrPattern32 &at, const CsrPattern32 *q, RsPlan &plan, cudaStream_t s,
             int ctas = 0);
// The packed words of a plan that a launch will use.
void rs_pack(const CsrPattern32 &a, const CsrPattern32 &at, const CsrPattern32 *q, RsPlan &plan, cudaStream_t s);

// f(a value of the index type of a launch): the plan's, or without its packing.
template <class F>
void rs_with_index(const RsPlan &plan, bool packed, F &&f) {
    if (packed)
        f(RsPacked());
    else if (plan.small)
        f(uint16_t());
    else
        f(int());
}
// CTAs (at most one per SM) and threads for `nnz` nonzeros. Timed per
// iteration (float64 Halpern, 37 / 74 / 148 CTAs x 256 / 512 / 768 / 1024
// threads): 4,000 nonzeros 4.6 us with 31 x 256 (148 x 1024: 5.3), 40,000
// nonzeros 5.2 us with 148 x 256 (37 x 256: 6.5, 148 x 1024: 5.5), 120,000
// nonzeros 6.0 us with 148 x 512 (256: 6.4, 1024: 6.5), 600,000 nonzeros 10.3
// us with 148 x 768 (256: 12.2, 1024: 10.9).
int rs_grid(int64_t nnz);
int rs_threads(int64_t nnz, int grid);

template <class K, class... A>
inline void rs_launch(K kernel, int grid, int threads, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(grid));
    cfg.blockDim = dim3(static_cast<unsigned>(threads));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    VK_CUDA(cudaLaunchKernelEx(&cfg, kernel, args...));
}

// True when `grid` CTAs of `kernel` are resident at once with `smem` bytes of
// dynamic shared memory each (also sets the kernel's shared-memory limit).
template <class K>
inline bool rs_fits(K kernel, int grid, int threads, size_t smem) {
    if (smem > static_cast<size_t>(kRsSmem)) return false;
    int dev = 0, sms = 0, per = 0, coop = 0;
    VK_CUDA(cudaGetDevice(&dev));
    VK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    VK_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    VK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kRsSmem));
    VK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, smem));
    return coop != 0 && grid <= per * sms;
}

} // namespace vk
