// Power iterations for the largest eigenvalues of many instances at once, the
// stopping rule on the device.
//
// A step is the passes of the operator (v <- M v / |v|, the division folded
// into a pass's epilogue as a factor, |M v|^2 summed in the last one) and one
// control kernel; the host looks at the number of unsettled instances every
// kPowerPoll steps instead of at every norm. An instance's estimate freezes at
// the step where it settles (or the last one allowed), so steps past it change
// nothing. With a host round trip, a norm by one block per instance and a scaling
// kernel per step, 200 steps took 12-15 ms on a 120,000-nonzero LP and 19 ms on
// 48 LPs of 2 million nonzeros.
#pragma once

#include "vk_csr.cuh"

namespace vk {

constexpr int kPowerSteps = 200; // at most
constexpr int kPowerPoll = 16;

struct PowerState {
    DevBuf<double> inv, est;      // 1 / |v| of the last step, estimates
    DevBuf<int> steps, unsettled; // steps per instance (negative once settled), instances still moving
    int count = 0;
};

// Starts `count` instances whose first vectors have the squared norms nrm2 (device).
void power_start(PowerState &p, int count, const double *nrm2, cudaStream_t s);
// One step's control: |M v|^2 of instance b = the sum of partials[begin[b] ..
// begin[b+1]) in a fixed order (begin null: one instance, `n` partials). The
// estimate is |M v| / |v|, its square root if `root`.
void power_control(PowerState &p, const double *partials, const int *begin, int n, bool root, cudaStream_t s);
// Runs step() until every instance has settled.
template <class F>
void power_run(PowerState &p, F &&step, cudaStream_t s) {
    int left = 1;
    for (int it = 0; left > 0 && it < kPowerSteps; ++it) {
        step();
        if (it % kPowerPoll != kPowerPoll - 1 && it != kPowerSteps - 1) continue;
        VK_CUDA(cudaMemcpyAsync(&left, p.unsettled.get(), sizeof(int), cudaMemcpyDeviceToHost, s));
        VK_CUDA(cudaStreamSynchronize(s));
    }
}

// y = s (times 1 / |v| when `inv` is given), and the sum of y^2 per warp-tile
// (TILES) or per CTA when `partials` is given. inst: instance of a row (null: 0).
template <bool TILES>
struct PowerEpi : EpiBase<double> {
    static constexpr int NR = 1;
    static constexpr bool kPerTile = TILES;
    double *y;
    const double *inv;
    const int *inst;
    double *partials;
    using Pre = typename EpiBase<double>::Pre;
    __device__ void row_pre(int i, const double (&s)[1], const Pre &, double (&red)[1]) const {
        const double v = inv ? s[0] * inv[inst ? inst[i] : 0] : s[0];
        y[i] = v;
        red[0] += v * v;
    }
    template <int R>
    __device__ void tile_done(int t, double (&red)[R]) const {
        if (partials) partials[t] = red[0];
    }
    __device__ void finish(double (&red)[1], double *scratch, int block) const {
        if (TILES || !partials) return;
        block_sum<1>(red, scratch);
        if (threadIdx.x == 0) partials[block] = red[0];
    }
};

} // namespace vk
