// The reference scheme on a resident LP (vk_resident.cuh): FAST-order iterations
// of vk_reference.cu, control steps included, `iterations` of them in one
// launch. Two grid barriers (2.7 us) bound an iteration of a small LP; the control
// step between them, which one thread takes while the GPU waits, has its norms
// on the way during the products, no division, and maxima by integer reductions:
// 2,000 x 5,000 LP 6.93 -> 5.92 us per iteration, 50,000 x 100,000 12.24 -> 10.87.
#pragma once

#include "vk_resident.cuh"
#include "vk_solver.h"

namespace vk {

// True when the control step of iteration k (which judges the metric of
// iteration k-1) may change tau / sigma or set the restart flag: pdhg.cpp:133,
// every 50 iterations after the first.
__device__ __forceinline__ bool ref_policy_iter(long long k) { return k >= 51 && (k - 1) % 50 == 0; }

// k % 50, counted along.
struct RefPhase {
    int at;
    __device__ explicit RefPhase(long long k) : at(static_cast<int>(k % 50)) {}
    __device__ void next() { at = at == 49 ? 0 : at + 1; }
    __device__ bool policy(long long k) const { return at == 1 && k >= 51; } // ref_policy_iter(k)
};

// The metric of iteration k-1 (c.rp, c.rd) and the step / restart / stop rules
// (pdhg.cpp:133-150). policy: ref_policy_iter(c.iter). A division is left to
// the steps that change sigma: one thread decides while a whole GPU waits.
__device__ inline void ref_decide(RefCtl &c, bool policy) {
    c.restart = 0; // consumed by the previous primal step (pdhg.cpp:98-100)
    if (c.iter >= 1) {
        const double metric = smax(c.rp, c.rd);
        c.last_metric = metric;
        if (policy) {
            if (metric > c.previous * 1.25) {
                c.tau *= 0.5;
                c.sigma *= 0.5;
                c.restart = 1;
                c.restarts += 1;
            } else if (metric < c.previous * 0.1) {
                c.tau = smin(c.tau * 1.05, c.max_step);
                c.sigma = c.tau;
            }
            c.inv_sigma = 1.0 / c.sigma;
            c.previous = metric;
        } else if (c.iter == 1) {
            c.previous = metric;
        }
        if (metric <= c.tol) {
            c.done = 1;
            c.status = VK_STATUS_OPTIMAL;
        }
    }
    if (!c.done && c.iter >= c.limit) {
        c.done = 1;
        c.status = VK_STATUS_ITERATION_LIMIT;
    }
    c.rp = 0.0;
    c.rd = 0.0;
}

// x_{k+1} from K'y (pdhg.cpp:92-97), the reference's roundings.
__device__ __forceinline__ double ref_primal(double tau, double aty, double x, double c, double l, double u) {
    const double t = __dadd_rn(__dmul_rn(-tau, c), x);
    return clampbox(__dadd_rn(__dmul_rn(-tau, aty), t), l, u);
}

struct RsRefArgs {
    const int *ro_a, *ci_a, *ro_t, *ci_t;
    const double *va, *vt;
    const int *part_a, *part_t;
    int cap_a, cap_t, rows, cols;
    double *x, *xn, *y, *kx; // x_k; x_{k+1} (gathered); y_k; K x_k
    const double *c, *l, *u, *rl, *ru;
    RefCtl *ctl;
    double *norms; // [2][4]: primal and stationarity norms by iteration (mod 4), zero at the launch
    unsigned *counter;
    int *err;
    int iterations;
    long long *cycles; // profiling: cycles of the column passes, control steps and row passes of CTA 0; else null
};

template <class I>
struct RsRefLayout {
    size_t va, vt, ia, it, roa, rot, prod, xs, ys, bytes;
    static constexpr int kXs = 6, kYs = 4; // own columns: x, x next, K'y, c, l, u; own rows: y, kx, rl, ru
    __host__ __device__ RsRefLayout(int cap_a, int cap_t, int rows, int cols) {
        size_t o = 0;
        const auto take = [&](size_t b) {
            const size_t at = o;
            o = (o + b + 15) & ~static_cast<size_t>(15);
            return at;
        };
        va = take(8 * static_cast<size_t>(cap_a));
        vt = take(8 * static_cast<size_t>(cap_t));
        ia = take(sizeof(I) * cap_a);
        it = take(sizeof(I) * cap_t);
        roa = take(4 * (static_cast<size_t>(rows) + 1));
        rot = take(4 * (static_cast<size_t>(cols) + 1));
        prod = take(8 * static_cast<size_t>(cap_a > cap_t ? cap_a : cap_t));
        xs = take(8 * kXs * static_cast<size_t>(cols));
        ys = take(8 * kYs * static_cast<size_t>(rows));
        bytes = o;
    }
};

template <class I>
__global__ void __launch_bounds__(kRsThreads, 1) rs_reference_kernel(RsRefArgs A) {
    extern __shared__ __align__(16) unsigned char rs_smem[];
    __shared__ RefCtl c;
    __shared__ double warps[32];
    if (A.ctl->done) return; // the same for the whole grid
    const int tid = threadIdx.x, nt = blockDim.x;
    const int r0 = A.part_a[blockIdx.x], rows = A.part_a[blockIdx.x + 1] - r0;
    const int c0 = A.part_t[blockIdx.x], cols = A.part_t[blockIdx.x + 1] - c0;
    const RsRefLayout<I> lay(A.cap_a, A.cap_t, A.rows, A.cols);
    const auto vec = [&](size_t o) { return reinterpret_cast<double *>(rs_smem + o); };
    const auto ind = [&](size_t o) { return reinterpret_cast<I *>(rs_smem + o); };
    const auto off = [&](size_t o) { return reinterpret_cast<int *>(rs_smem + o); };
    double *prod = vec(lay.prod);
    double *x = vec(lay.xs), *xn = x + A.cols, *aty = xn + A.cols, *cc = aty + A.cols, *l = cc + A.cols, *u = l + A.cols;
    double *y = vec(lay.ys), *kx = y + A.rows, *rl = kx + A.rows, *ru = rl + A.rows;
    RsBarrier bar{A.counter, A.err};
    if (tid == 0) c = *A.ctl;
    const auto sa = rs_load<double, I>(A.ro_a, A.ci_a, A.va, r0, r0 + rows, vec(lay.va), ind(lay.ia), off(lay.roa));
    const auto st = rs_load<double, I>(A.ro_t, A.ci_t, A.vt, c0, c0 + cols, vec(lay.vt), ind(lay.it), off(lay.rot));
    for (int j = tid; j < cols; j += nt) {
        x[j] = A.x[c0 + j];
        cc[j] = A.c[c0 + j];
        l[j] = A.l[c0 + j];
        u[j] = A.u[c0 + j];
    }
    for (int i = tid; i < rows; i += nt) {
        y[i] = A.y[r0 + i];
        kx[i] = A.kx[r0 + i];
        rl[i] = A.rl[r0 + i];
        ru[i] = A.ru[r0 + i];
    }
    __syncthreads();
    double *rp = A.norms, *rd = A.norms + 4;
    const long long start = c.iter, end = start + A.iterations;
    RefPhase phase(start);
    long long *const cycles = blockIdx.x == 0 && tid == 0 ? A.cycles : nullptr;
    long long mark = cycles ? clock64() : 0;
    const auto lap = [&](int q) {
        if (!cycles) return;
        const long long now = clock64();
        cycles[q] += now - mark;
        mark = now;
    };
    struct ColIn {
        double x, c, l, u;
    };
    struct RowIn {
        double y, kx, lo, hi;
    };
    for (long long k = start;; ++k, phase.next()) {
        // K'y_k, the stationarity of iteration k-1, and the primal step of
        // iteration k unless the control step may still change tau
        const bool policy = phase.policy(k);
        const double tau = c.tau;
        rs_products(st, A.y, prod);
        double top = 0.0;
        const auto column = [&](int j) { return ColIn{x[j], cc[j], l[j], u[j]}; };
        rs_rows(st, prod, column, [&](int j, double sum, const ColIn &p) {
            if (policy)
                aty[j] = sum;
            else
                A.xn[c0 + j] = xn[j] = ref_primal(tau, sum, p.x, p.c, p.l, p.u);
            if (k >= 1) {
                const double px = clampbox(__dadd_rn(-__dadd_rn(sum, p.c), p.x), p.l, p.u);
                top = smax(top, fabs(__dadd_rn(-px, p.x)));
            }
        });
        if (!bar.sync_max(top, warps, rd + (k & 3))) return;
        lap(0);
        // control: every CTA from the same numbers
        if (k == end) { // this launch ends here; the next one repeats the column pass
            if (blockIdx.x == 0 && tid == 0) {
                c.rp = __ldcg(rp + ((k - 1) & 3));
                *A.ctl = c;
            }
            break;
        }
        if (policy) {
            if (tid == 0) {
                if (k > start) c.rp = __ldcg(rp + ((k - 1) & 3));
                c.rd = __ldcg(rd + (k & 3));
                ref_decide(c, policy);
            }
            __syncthreads();
            for (int j = tid; j < cols; j += nt) A.xn[c0 + j] = xn[j] = ref_primal(c.tau, aty[j], x[j], cc[j], l[j], u[j]);
            if (!bar.sync()) return;
        }
        lap(1);
        double norm_p = 0.0, norm_d = 0.0; // on their way while the products are
        if (!policy && tid == 0) {
            norm_p = __ldcg(rp + ((k - 1) & 3));
            norm_d = __ldcg(rd + (k & 3));
        }
        rs_products(sa, A.xn, prod);
        if (!policy && tid == 0) {
            if (k > start) c.rp = norm_p;
            c.rd = norm_d;
            ref_decide(c, policy);
        }
        __syncthreads(); // c
        if (c.done) { // x_k, y_k are the answer
            if (blockIdx.x == 0 && tid == 0) *A.ctl = c;
            break;
        }
        // the slots of iteration k + 2: last read before this iteration's first barrier
        if (blockIdx.x == 0 && tid == 0) rp[(k + 2) & 3] = rd[(k + 2) & 3] = 0.0;
        const double sigma = c.sigma, inv = c.inv_sigma;
        const bool restart = c.restart != 0;
        top = 0.0;
        const auto dual = [&](int i) { return RowIn{y[i], kx[i], rl[i], ru[i]}; };
        rs_rows(sa, prod, dual, [&](int i, double kxn, const RowIn &p) {
            const double kxbar = restart ? kxn : __dadd_rn(__dmul_rn(2.0, kxn), -p.kx);
            const double yarg = __dadd_rn(__dmul_rn(sigma, kxbar), p.y);
            const double yp = clampbox(__dmul_rn(inv, yarg), p.lo, p.hi);
            A.y[r0 + i] = y[i] = __dadd_rn(__dmul_rn(-sigma, yp), yarg);
            kx[i] = kxn;
            top = smax(top, fabs(__dadd_rn(clampbox(kxn, p.lo, p.hi), -kxn)));
        });
        if (!bar.sync_max(top, warps, rp + (k & 3))) return;
        lap(2);
        if (tid == 0) c.iter += 1;
        double *t = x;
        x = xn;
        xn = t;
        __syncthreads();
    }
    for (int j = tid; j < cols; j += nt) A.x[c0 + j] = x[j];
    for (int i = tid; i < rows; i += nt) A.kx[r0 + i] = kx[i];
}

} // namespace vk
