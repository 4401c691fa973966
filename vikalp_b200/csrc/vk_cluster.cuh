// An LP in one thread-block cluster.
//
// For the smallest LPs even the grid barrier of the resident kernels
// (vk_resident.cuh, 2,500 cycles a pass) is most of an iteration. Here eight CTAs
// on neighbouring SMs hold the matrices (16-bit indices) and a full copy of both
// gathered vectors in shared memory: a gather is a local load, each new entry
// is stored into all eight copies (distributed shared memory) and the cluster's
// hardware barrier (700 cycles) orders the passes; nothing goes to L2 until the
// launch ends. A CTA overwrites the vector of a pass only two passes later, past
// a barrier that every CTA reaches after its last read of it. All CTAs take the
// same decisions from the same numbers, so they meet at the same barriers.
//
// The copies cross at about 15 bytes per cycle and SM, so that LPs with longer
// vectors are faster resident in the whole GPU: kClVectorBytes, measured beside
// the Halpern kernel (vk_halpern_cluster.cuh).
#pragma once

#include "vk_resident.cuh"

namespace vk {

constexpr int kClRanks = 8;                // CTAs of the cluster (the portable maximum)
constexpr int kClThreads = 512;            // threads of a CTA, at most
constexpr size_t kClVectorBytes = 32 << 10; // the two gathered vectors together

// Byte offsets in a CTA's dynamic shared memory; XS / YS: the vectors it keeps of
// its own columns / rows.
template <class T, int XS, int YS>
struct ClLayout {
    size_t xf, yf, va, vt, ia, it, roa, rot, xs, ys, bytes;
    __host__ __device__ ClLayout(int m, int n, int cap_a, int cap_t, int rows, int cols) {
        size_t o = 0;
        const auto take = [&](size_t b) {
            const size_t at = o;
            o = (o + b + 15) & ~static_cast<size_t>(15);
            return at;
        };
        xf = take(sizeof(T) * n);
        yf = take(sizeof(T) * m);
        va = take(sizeof(T) * cap_a);
        vt = take(sizeof(T) * cap_t);
        ia = take(2 * static_cast<size_t>(cap_a));
        it = take(2 * static_cast<size_t>(cap_t));
        roa = take(4 * (static_cast<size_t>(rows) + 1));
        rot = take(4 * (static_cast<size_t>(cols) + 1));
        xs = take(sizeof(T) * XS * static_cast<size_t>(cols));
        ys = take(sizeof(T) * YS * static_cast<size_t>(rows));
        bytes = o;
    }
};

// Every thread of the cluster; shared-memory writes before it, remote ones
// included, are visible after it.
__device__ __forceinline__ void cl_sync() {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ int cl_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return static_cast<int>(r);
}
// The address, in rank p's shared memory, of this CTA's shared variable at `local`.
__device__ __forceinline__ uint32_t cl_map(uint32_t local, int p) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local), "r"(p));
    return a;
}
__device__ __forceinline__ void cl_store(uint32_t addr, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
__device__ __forceinline__ void cl_store(uint32_t addr, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
// vec[i] = v in every rank's copy; the L lanes that hold v share the ranks.
template <class T>
__device__ __forceinline__ void cl_put(T *vec, int i, T v, int sl, int L) {
    const uint32_t a = smem_u32(vec + i);
    for (int p = sl; p < kClRanks; p += L) cl_store(cl_map(a, p), v);
}

// row(r, sum, pre(r), lane, L) for every row in every lane of its group of L,
// sum = sum_k v_k x[idx_k] with x in shared memory; A: the sums' type (float64
// in the checks).
template <class A, class T, class P, class F>
__device__ __forceinline__ void cl_pass(const RsSide<T, uint16_t> &s, const T *x, P &&pre, F &&row) {
    const int L = s.L, lane = threadIdx.x & 31, sl = lane & (L - 1);
    const int first = (static_cast<int>(threadIdx.x) & ~31) / L; // the warp's first row: uniform trip count
    for (int rb = first; rb < s.rows; rb += static_cast<int>(blockDim.x) / L) {
        const int r = rb + lane / L;
        const bool valid = r < s.rows;
        decltype(pre(0)) in{};
        A acc = A(0);
        if (valid) {
            in = pre(r);
            const int b = s.ro[r + 1];
            for (int k = s.ro[r] + sl; k < b; k += L) acc += static_cast<A>(s.v[k]) * static_cast<A>(x[s.idx[k]]);
        }
        acc = rs_group_sum(acc, L);
        __syncwarp(); // every lane has its inputs before the lead lane updates them
        if (valid) row(r, acc, in, sl, L);
    }
}

// Whether a cluster of `kernel` can run with `bytes` of dynamic shared memory in
// each CTA (allowed from here on).
template <class K>
bool cl_fits(K *kernel, int threads, size_t bytes) {
    if (bytes > static_cast<size_t>(kRsSmem)) return false;
    VK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kRsSmem));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(kClRanks);
    cfg.blockDim = dim3(static_cast<unsigned>(threads));
    cfg.dynamicSmemBytes = bytes;
    int clusters = 0;
    VK_CUDA(cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg));
    return clusters > 0;
}
// Threads of a CTA: 300 x 800 LP with 4,000 nonzeros 2.42 us per Halpern
// iteration with 256 (512: 2.45), 1,000 x 2,000 with 16,000 3.70 with 512 (3.90).
inline int cl_threads(long long nnz) { return nnz <= 8192 ? 256 : kClThreads; }

} // namespace vk
