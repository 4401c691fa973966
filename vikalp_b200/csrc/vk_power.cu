// Control kernels of the power iterations (vk_power.cuh).
#include "vk_power.cuh"

namespace vk {

namespace {
constexpr int kThreads = 256;

__global__ void start_kernel(int count, const double *__restrict__ nrm2, double *__restrict__ inv,
                             double *__restrict__ est, int *__restrict__ steps, int *__restrict__ unsettled) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= count) return;
    inv[b] = nrm2[b] > 0.0 ? 1.0 / sqrt(nrm2[b]) : 1.0;
    est[b] = 0.0;
    steps[b] = 0;
    if (b == 0) *unsettled = count;
}

// One block per instance.
__global__ void __launch_bounds__(kThreads)
    control_kernel(const double *__restrict__ partials, const int *__restrict__ begin, int n, bool root,
                   double *__restrict__ inv, double *__restrict__ est, int *__restrict__ steps,
                   int *__restrict__ unsettled) {
    __shared__ double scratch[32];
    const int b = blockIdx.x;
    const int t0 = begin ? begin[b] : 0, t1 = begin ? begin[b + 1] : n;
    double s[1] = {0.0};
    for (int t = t0 + static_cast<int>(threadIdx.x); t < t1; t += kThreads) s[0] += partials[t];
    block_sum<1>(s, scratch);
    if (threadIdx.x != 0) return;
    const double nz = sqrt(s[0]);
    inv[b] = s[0] > 0.0 ? 1.0 / nz : 1.0;
    const int it = steps[b];
    if (it < 0) return; // settled
    const double e = root ? sqrt(nz) : nz;
    const bool done = it > 10 && fabs(e - est[b]) <= 1e-6 * e;
    est[b] = e;
    steps[b] = done ? -1 : it + 1;
    if (done) atomicSub(unsettled, 1);
}
} // namespace

void power_start(PowerState &p, int count, const double *nrm2, cudaStream_t s) {
    p.count = count;
    p.inv.reset(count);
    p.est.reset(count);
    p.steps.reset(count);
    p.unsettled.reset(1);
    start_kernel<<<ceil_div(count, kThreads), kThreads, 0, s>>>(count, nrm2, p.inv.get(), p.est.get(), p.steps.get(),
                                                                p.unsettled.get());
    VK_LAUNCH_CHECK();
}

void power_control(PowerState &p, const double *partials, const int *begin, int n, bool root, cudaStream_t s) {
    control_kernel<<<p.count, kThreads, 0, s>>>(partials, begin, n, root, p.inv.get(), p.est.get(), p.steps.get(),
                                                p.unsettled.get());
    VK_LAUNCH_CHECK();
}

} // namespace vk
