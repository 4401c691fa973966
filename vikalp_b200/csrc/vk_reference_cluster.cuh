// The reference scheme on an LP in one thread-block cluster (vk_cluster.cuh):
// the iterations of vk_reference_resident.cuh, control steps included,
// `iterations` of them in one launch. Microseconds per iteration: 5 x 8 LP 2.36,
// 300 x 800 2.92, 1,000 x 2,000 with 16,000 nonzeros 4.12, 1,300 x 2,700 with
// 32,400 5.35 (with the division and the shuffled maxima that the control step
// had before, 3.07, 3.62, 4.63 and 5.95 against 5.56, 6.19, 6.36 and 6.82 of the
// resident kernel, which has since gained a microsecond too).
#pragma once

#include "vk_cluster.cuh"
#include "vk_reference_resident.cuh"

namespace vk {

// own columns: x, x next, K'y, c, l, u; own rows: y, kx, rl, ru
using ClRefLayout = ClLayout<double, 6, 4>;

// The warp's maximum of v >= 0, left in this warp's
// slot in every rank's copy.
__device__ __forceinline__ void cl_put_max(double v, double (*slots)[kClThreads / 32], int rank) {
    const int lane = threadIdx.x & 31;
    v = rs_warp_max(v);
    if (lane < kClRanks) cl_store(cl_map(smem_u32(&slots[rank][threadIdx.x >> 5]), lane), v);
}
// The lane's part of the maximum over all slots.
__device__ __forceinline__ double cl_part_max(const double (*slots)[kClThreads / 32]) {
    double v = 0.0;
#pragma unroll
    for (int i = 0; i < kClRanks * (kClThreads / 32); i += 32) v = smax(v, (&slots[0][0])[i + (threadIdx.x & 31)]);
    return v;
}

__global__ void __cluster_dims__(kClRanks, 1, 1) __launch_bounds__(kClThreads, 1)
    cl_reference_kernel(RsRefArgs A, int m, int n) {
    extern __shared__ __align__(16) unsigned char cl_smem[];
    __shared__ RefCtl c;
    // row passes alternate between two sets: a rank may be in its next row pass
    // while another still reads the last one's maxima
    __shared__ double prim[2][kClRanks][kClThreads / 32], stat[kClRanks][kClThreads / 32];
    if (A.ctl->done) return; // the same for the whole cluster
    const int rank = cl_rank(), tid = threadIdx.x, nt = blockDim.x;
    const int r0 = A.part_a[rank], rows = A.part_a[rank + 1] - r0;
    const int c0 = A.part_t[rank], cols = A.part_t[rank + 1] - c0;
    const ClRefLayout lay(m, n, A.cap_a, A.cap_t, A.rows, A.cols);
    const auto vec = [&](size_t o) { return reinterpret_cast<double *>(cl_smem + o); };
    const auto ind = [&](size_t o) { return reinterpret_cast<uint16_t *>(cl_smem + o); };
    const auto off = [&](size_t o) { return reinterpret_cast<int *>(cl_smem + o); };
    double *xf = vec(lay.xf), *yf = vec(lay.yf);
    double *x = vec(lay.xs), *xn = x + A.cols, *aty = xn + A.cols, *cc = aty + A.cols, *l = cc + A.cols, *u = l + A.cols;
    double *y = vec(lay.ys), *kx = y + A.rows, *rl = kx + A.rows, *ru = rl + A.rows;
    if (tid == 0) c = *A.ctl;
    const auto sa = rs_load<double, uint16_t>(A.ro_a, A.ci_a, A.va, r0, r0 + rows, vec(lay.va), ind(lay.ia), off(lay.roa));
    const auto st = rs_load<double, uint16_t>(A.ro_t, A.ci_t, A.vt, c0, c0 + cols, vec(lay.vt), ind(lay.it), off(lay.rot));
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
    for (int i = tid; i < m; i += nt) yf[i] = A.y[i];
    for (int i = tid; i < kClRanks * (kClThreads / 32); i += nt) // with fewer warps, the rest stay 0
        (&stat[0][0])[i] = (&prim[0][0][0])[i] = (&prim[1][0][0])[i] = 0.0;
    cl_sync(); // every rank has started (remote stores may reach it) and is loaded
    const long long start = c.iter, end = start + A.iterations;
    RefPhase phase(start);
    long long *const cycles = rank == 0 && tid == 0 ? A.cycles : nullptr;
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
        double top = 0.0;
        const auto column = [&](int j) { return ColIn{x[j], cc[j], l[j], u[j]}; };
        cl_pass<double>(st, yf, column, [&](int j, double sum, const ColIn &p, int sl, int L) {
            if (policy) {
                if (sl == 0) aty[j] = sum;
            } else {
                const double v = ref_primal(tau, sum, p.x, p.c, p.l, p.u);
                cl_put(xf, c0 + j, v, sl, L);
                if (sl == 0) xn[j] = v;
            }
            if (k >= 1) {
                const double px = clampbox(__dadd_rn(-__dadd_rn(sum, p.c), p.x), p.l, p.u);
                top = smax(top, fabs(__dadd_rn(-px, p.x)));
            }
        });
        cl_put_max(top, stat, rank);
        cl_sync();
        lap(0);
        // control: every rank from the same numbers
        if (tid < 32) {
            // (the decision takes the larger of the two norms; the launch's last
            // step keeps the primal one, its column pass will be repeated)
            double v = cl_part_max(prim[(k + 1) & 1]);
            if (k < end) v = smax(v, cl_part_max(stat));
            v = rs_warp_max(v);
            if (tid == 0) {
                if (k == start)
                    c.rd = v;
                else
                    c.rp = v;
                if (k < end) ref_decide(c, policy);
            }
        }
        __syncthreads();
        if (k == end || c.done) break; // x_k, y_k; the next launch, if any, repeats the column pass
        if (policy) {
            for (int j = tid; j < cols; j += nt) {
                const double v = ref_primal(c.tau, aty[j], x[j], cc[j], l[j], u[j]);
                xn[j] = v;
                cl_put(xf, c0 + j, v, 0, 1);
            }
            cl_sync();
        }
        lap(1);
        const double sigma = c.sigma, inv = c.inv_sigma;
        const bool restart = c.restart != 0;
        top = 0.0;
        const auto dual = [&](int i) { return RowIn{y[i], kx[i], rl[i], ru[i]}; };
        cl_pass<double>(sa, xf, dual, [&](int i, double kxn, const RowIn &p, int sl, int L) {
            const double kxbar = restart ? kxn : __dadd_rn(__dmul_rn(2.0, kxn), -p.kx);
            const double yarg = __dadd_rn(__dmul_rn(sigma, kxbar), p.y);
            const double yp = clampbox(__dmul_rn(inv, yarg), p.lo, p.hi);
            const double yn = __dadd_rn(__dmul_rn(-sigma, yp), yarg);
            cl_put(yf, r0 + i, yn, sl, L);
            if (sl == 0) {
                y[i] = yn;
                kx[i] = kxn;
            }
            top = smax(top, fabs(__dadd_rn(clampbox(kxn, p.lo, p.hi), -kxn)));
        });
        cl_put_max(top, prim[k & 1], rank);
        cl_sync();
        lap(2);
        if (tid == 0) c.iter += 1; // read again past the next barrier
        double *t = x;
        x = xn;
        xn = t;
    }
    for (int j = tid; j < cols; j += nt) A.x[c0 + j] = x[j];
    for (int i = tid; i < rows; i += nt) {
        A.y[r0 + i] = y[i];
        A.kx[r0 + i] = kx[i];
    }
    if (rank == 0 && tid == 0) *A.ctl = c;
}

} // namespace vk
