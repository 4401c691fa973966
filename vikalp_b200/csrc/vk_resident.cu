// Host side of the resident iterations (vk_resident.cuh).
#include "vk_resident.cuh"

namespace vk {

namespace {
// Boundaries of `rows` rows over `ctas` shares of about equal cost.
std::vector<int> partition(const std::vector<int> &ro, int rows, int ctas) {
    std::vector<int> at(static_cast<size_t>(ctas) + 1, rows);
    at[0] = 0;
    const auto cost = [&](int r) { return static_cast<int64_t>(ro[r]) + static_cast<int64_t>(kRsRowCost) * r; };
    const int64_t total = cost(rows);
    for (int b = 1; b < ctas; ++b) {
        int lo = at[b - 1], hi = rows; // the first row at or past the share's start
        while (lo < hi) {
            const int mid = (lo + hi) / 2;
            if (cost(mid) * ctas < total * b)
                lo = mid + 1;
            else
                hi = mid;
        }
        at[b] = lo;
    }
    return at;
}

int largest_share(const std::vector<int> &ro, const std::vector<int> &at) {
    int most = 0;
    for (size_t b = 0; b + 1 < at.size(); ++b) most = std::max(most, ro[at[b + 1]] - ro[at[b]]);
    return most;
}

int most_rows(const std::vector<int> &at) {
    int most = 0;
    for (size_t b = 0; b + 1 < at.size(); ++b) most = std::max(most, at[b + 1] - at[b]);
    return most;
}
constexpr int kRsPlaces = 1 << RsPacked::kPlaceBits;

// out: the RsPacked words of every share, in column order (places ascending
// within a column). One CTA sorts a share in shared memory (bitonic): about 25 us
// for 600,000 nonzeros, once per handle; sorted again by every launch it had cost
// the solves of less than 64 iterations more than the order gave them.
__global__ void __launch_bounds__(1024) rs_pack_kernel(const int *__restrict__ ro, const int *__restrict__ ci,
                                                       const int *__restrict__ part, int count, int *__restrict__ out) {
    extern __shared__ uint32_t key[]; // count: a power of two, at least the share
    const int k0 = ro[part[blockIdx.x]], nnz = ro[part[blockIdx.x + 1]] - k0;
    for (int k = threadIdx.x; k < count; k += blockDim.x)
        key[k] = k < nnz ? static_cast<uint32_t>(ci[k0 + k]) << RsPacked::kPlaceBits | static_cast<uint32_t>(k)
                         : 0xffffffffu; // not below any word
    for (int size = 2; size <= count; size <<= 1)
        for (int gap = size >> 1; gap > 0; gap >>= 1) {
            __syncthreads();
            for (int t = threadIdx.x; t < count / 2; t += blockDim.x) {
                const int a = 2 * t - (t & (gap - 1)), b = a + gap;
                const uint32_t ka = key[a], kb = key[b];
                if ((ka > kb) == ((a & size) == 0)) {
                    key[a] = kb;
                    key[b] = ka;
                }
            }
        }
    __syncthreads();
    for (int k = threadIdx.x; k < nnz; k += blockDim.x) out[k0 + k] = static_cast<int>(key[k]);
}

void pack(const CsrPattern32 &p, const DevBuf<int> &part, int grid, int cap, DevBuf<int> &out, cudaStream_t s) {
    out.reset(std::max<int64_t>(p.nnz, 1));
    int count = 2;
    while (count < cap) count *= 2;
    rs_pack_kernel<<<grid, std::min(1024, std::max(32, count / 2)), count * sizeof(uint32_t), s>>>(
        p.ro.get(), p.ci.get(), part.get(), count, out.get());
    VK_LAUNCH_CHECK();
}
} // namespace

bool rs_plan(const CsrPattern32 &a, const CsrPattern32 &at, const CsrPattern32 *q, RsPlan &plan, cudaStream_t s,
             int ctas) {
    if (a.rows == 0 || a.nnz == 0 || forced_variant() >= 0) return false;
    const int64_t stored = 2 * a.nnz + (q ? q->nnz : 0);
    if (stored * static_cast<int64_t>(sizeof(float) + 2) > static_cast<int64_t>(kRsMaxGrid) * kRsSmem) return false;
    const int m = a.rows, n = a.cols;
    std::vector<int> ro(m + 1), rot(n + 1), roq(q ? n + 1 : 0);
    VK_CUDA(cudaMemcpyAsync(ro.data(), a.ro.get(), ro.size() * sizeof(int), cudaMemcpyDeviceToHost, s));
    VK_CUDA(cudaMemcpyAsync(rot.data(), at.ro.get(), rot.size() * sizeof(int), cudaMemcpyDeviceToHost, s));
    if (q) VK_CUDA(cudaMemcpyAsync(roq.data(), q->ro.get(), roq.size() * sizeof(int), cudaMemcpyDeviceToHost, s));
    VK_CUDA(cudaStreamSynchronize(s));
    plan.grid = ctas > 0 ? ctas : rs_grid(a.nnz);
    plan.threads = rs_threads(a.nnz, plan.grid);
    plan.small = m <= 65536 && n <= 65536;
    // columns are split by their nonzeros in A and Q together
    std::vector<int> both(rot);
    for (size_t j = 0; j < roq.size(); ++j) both[j] += roq[j];
    const std::vector<int> pa = partition(ro, m, plan.grid), pt = partition(both, n, plan.grid);
    plan.rows = most_rows(pa);
    plan.cols = most_rows(pt);
    plan.cap_a = largest_share(ro, pa);
    plan.cap_t = largest_share(rot, pt);
    plan.cap_q = q ? largest_share(roq, pt) : 0;
    plan.part_a.reset(pa.size());
    plan.part_t.reset(pt.size());
    plan.counter.reset(1);
    VK_CUDA(cudaMemcpyAsync(plan.part_a.get(), pa.data(), plan.part_a.bytes(), cudaMemcpyHostToDevice, s));
    VK_CUDA(cudaMemcpyAsync(plan.part_t.get(), pt.data(), plan.part_t.bytes(), cudaMemcpyHostToDevice, s));
    // column order: a plan for the whole GPU whose columns and shares fit the bits
    constexpr int kCols = 1 << RsPacked::kColBits;
    const int most = std::max({plan.cap_a, plan.cap_t, plan.cap_q});
    plan.packed = ctas == 0 && m <= kCols && n <= kCols && most <= kRsPlaces;
    VK_CUDA(cudaStreamSynchronize(s)); // the boundaries live on this stack frame
    return true;
}

void rs_pack(const CsrPattern32 &a, const CsrPattern32 &at, const CsrPattern32 *q, RsPlan &plan, cudaStream_t s) {
    pack(a, plan.part_a, plan.grid, plan.cap_a, plan.words_a, s);
    pack(at, plan.part_t, plan.grid, plan.cap_t, plan.words_t, s);
    if (q) pack(*q, plan.part_t, plan.grid, plan.cap_q, plan.words_q, s);
}

int rs_grid(int64_t nnz) {
    int dev = 0, sms = 0;
    VK_CUDA(cudaGetDevice(&dev));
    VK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    return std::min(std::min(sms, kRsMaxGrid), std::max(1, static_cast<int>(nnz / 128)));
}

int rs_threads(int64_t nnz, int grid) {
    const int64_t share = nnz / grid;
    return share <= 512 ? 256 : share <= 1024 ? 512 : 768;
}

} // namespace vk
