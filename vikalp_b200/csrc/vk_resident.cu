// Host side of the resident iterations (vk_resident.cuh).
#include "vk_resident.cuh"

namespace vk {

RsPart rs_partition(const std::vector<int> &ro, int rows, int ctas) {
    RsPart p;
    p.at.assign(static_cast<size_t>(ctas) + 1, rows);
    p.at[0] = 0;
    const auto cost = [&](int r) { return static_cast<int64_t>(ro[r]) + static_cast<int64_t>(kRsRowCost) * r; };
    const int64_t total = cost(rows);
    for (int b = 1; b < ctas; ++b) {
        int lo = p.at[b - 1], hi = rows; // the first row at or past the share's start
        while (lo < hi) {
            const int mid = (lo + hi) / 2;
            if (cost(mid) * ctas < total * b)
                lo = mid + 1;
            else
                hi = mid;
        }
        p.at[b] = lo;
    }
    for (int b = 0; b < ctas; ++b) {
        p.rows = std::max(p.rows, p.at[b + 1] - p.at[b]);
        p.nnz = std::max<int64_t>(p.nnz, ro[p.at[b + 1]] - ro[p.at[b]]);
    }
    return p;
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
