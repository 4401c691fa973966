// The restarted Halpern scheme on an LP in one thread-block cluster: the
// iterations, checks and restarts of vk_halpern.cu, `chunks` check intervals in
// one launch.
//
// Microseconds per iteration, float64, against the resident kernel: 5 x 8 LP
// 1.74 (3.56), 300 x 800 2.64 (4.92), 1,000 x 2,000 with 16,000 nonzeros 3.60
// (5.12), 1,300 x 2,700 with 21,600 4.43 (5.06); with many nonzeros, 1,300 x 2,700
// with 32,400 4.71 (5.33), 1,000 x 2,000 with 60,000 5.35 (5.89), 200 x 400 with
// 48,000 3.39 (5.32). The copies cross at about 15
// bytes per cycle and SM, so that longer vectors lose: 1,600 x 3,400 with 27,200
// 5.09 (5.03), 2,000 x 4,100 6.28 (5.09). Hence kClVectorBytes.
#pragma once

#include "vk_cluster.cuh"
#include "vk_halpern_resident.cuh"

namespace vk {

// own columns: x, x0, c, l, u; own rows: y, y0, rl, ru
template <class T>
using ClHalLayout = ClLayout<T, 5, 4>;

template <class T>
__global__ void __cluster_dims__(kClRanks, 1, 1) __launch_bounds__(kClThreads, 1)
    cl_halpern_kernel(RsHalArgs<T> A, int m, int n) {
    extern __shared__ __align__(16) unsigned char cl_smem[];
    __shared__ HalCtl c;
    __shared__ double slots[kClRanks][kCheckSums], scratch[32 * kCheckSums];
    if (A.ctl->done) return; // the same for the whole cluster
    const int rank = cl_rank(), tid = threadIdx.x, nt = blockDim.x;
    const int r0 = A.part_a[rank], rows = A.part_a[rank + 1] - r0;
    const int c0 = A.part_t[rank], cols = A.part_t[rank + 1] - c0;
    const ClHalLayout<T> lay(m, n, A.cap_a, A.cap_t, A.rows, A.cols);
    const auto vec = [&](size_t o) { return reinterpret_cast<T *>(cl_smem + o); };
    const auto ind = [&](size_t o) { return reinterpret_cast<uint16_t *>(cl_smem + o); };
    const auto off = [&](size_t o) { return reinterpret_cast<int *>(cl_smem + o); };
    T *xf = vec(lay.xf), *yf = vec(lay.yf);
    T *x = vec(lay.xs), *x0 = x + A.cols, *cc = x0 + A.cols, *l = cc + A.cols, *u = l + A.cols;
    T *y = vec(lay.ys), *y0 = y + A.rows, *rl = y0 + A.rows, *ru = rl + A.rows;
    if (tid == 0) c = *A.ctl;
    const auto sa = rs_load<T, uint16_t>(A.ro_a, A.ci_a, A.va, r0, r0 + rows, vec(lay.va), ind(lay.ia), off(lay.roa));
    const auto st = rs_load<T, uint16_t>(A.ro_t, A.ci_t, A.vt, c0, c0 + cols, vec(lay.vt), ind(lay.it), off(lay.rot));
    for (int j = tid; j < cols; j += nt) {
        x[j] = A.x[c0 + j];
        x0[j] = A.x0[c0 + j];
        cc[j] = A.c[c0 + j];
        l[j] = A.l[c0 + j];
        u[j] = A.u[c0 + j];
    }
    for (int i = tid; i < rows; i += nt) {
        y[i] = A.y[r0 + i];
        y0[i] = A.y0[r0 + i];
        rl[i] = A.rl[r0 + i];
        ru[i] = A.ru[r0 + i];
    }
    for (int i = tid; i < m; i += nt) yf[i] = A.y[i];
    cl_sync(); // every rank has started (remote stores may reach it) and is loaded

    struct ColIn {
        T x, x0, c, l, u;
    };
    struct RowIn {
        T y, y0, lo, hi;
    };
    for (int ch = 0; ch < A.chunks; ++ch) {
        const T tau = static_cast<T>(c.tau), sigma = static_cast<T>(c.sigma), rho = static_cast<T>(c.rho);
        const double kb = static_cast<double>(c.k_base);
        double s[kCheckSums];
#pragma unroll
        for (int r = 0; r < kCheckSums; ++r) s[r] = 0.0;
        for (int it = 0; it < A.chunk; ++it) {
            const double k = kb + it;
            const T lam = static_cast<T>((k + 1.0) / (k + 2.0));
            const bool check = it == A.chunk - 1;
            const auto column = [&](int j) { return ColIn{x[j], x0[j], cc[j], l[j], u[j]}; };
            cl_pass<T>(st, yf, column, [&](int j, T sum, const ColIn &p, int sl, int L) {
                const T xh = clampbox(p.x - tau * (p.c + sum), p.l, p.u);
                cl_put(xf, c0 + j, T(2) * xh - p.x, sl, L);
                if (sl != 0) return;
                x[j] = lam * ((T(1) + rho) * xh - rho * p.x) + (T(1) - lam) * p.x0;
                if (check) {
                    A.xhat[c0 + j] = xh;
                    const double d0 = static_cast<double>(xh) - static_cast<double>(p.x);
                    const double d1 = static_cast<double>(xh) - static_cast<double>(p.x0);
                    s[0] += d0 * d0;
                    s[1] += d1 * d1;
                }
            });
            cl_sync();
            const auto dual = [&](int i) { return RowIn{y[i], y0[i], rl[i], ru[i]}; };
            cl_pass<T>(sa, xf, dual, [&](int i, T sum, const RowIn &p, int sl, int L) {
                const T v = p.y + sigma * sum;
                const T yh = v - clampbox(v, sigma * p.lo, sigma * p.hi);
                const T yn = lam * ((T(1) + rho) * yh - rho * p.y) + (T(1) - lam) * p.y0;
                cl_put(yf, r0 + i, yn, sl, L);
                if (sl != 0) return;
                y[i] = yn;
                if (check) {
                    A.yhat[r0 + i] = yh;
                    const double d0 = static_cast<double>(yh) - static_cast<double>(p.y);
                    const double d1 = static_cast<double>(yh) - static_cast<double>(p.y0);
                    s[2] += d0 * d0;
                    s[3] += d1 * d1;
                }
            });
            cl_sync();
        }
        // the check: (x^, y^) into the gathered vectors, K x^ and K'y^
        for (int j = tid; j < cols; j += nt) cl_put(xf, c0 + j, A.xhat[c0 + j], 0, 1);
        for (int i = tid; i < rows; i += nt) cl_put(yf, r0 + i, A.yhat[r0 + i], 0, 1);
        cl_sync();
        const auto none = [](int) { return 0; };
        cl_pass<double>(sa, xf, none, [&](int i, double sum, int, int sl, int) {
            if (sl == 0) kkt_row_terms(sum, rl[i], ru[i], A.rs[r0 + i], yf[r0 + i], s + kColCheckSums + kRowCheckSums);
        });
        cl_pass<double>(st, yf, none, [&](int j, double sum, int, int sl, int) {
            if (sl == 0)
                kkt_col_terms(sum, cc[j], 0.0, A.cs[c0 + j], l[j], u[j], xf[c0 + j], s + kCheckSums - kKktColSums);
        });
        // the sums of all ranks, added in rank order by every rank
        block_sum<kCheckSums>(s, scratch); // the block's, in every lane of warp 0
        if (tid < kClRanks) {
            const uint32_t to = cl_map(smem_u32(&slots[rank][0]), tid);
#pragma unroll
            for (int r = 0; r < kCheckSums; ++r) cl_store(to + 8 * r, s[r]);
        }
        cl_sync();
        if (tid == 0) {
            for (int r = 0; r < kCheckSums; ++r) {
                s[r] = 0.0;
                for (int p = 0; p < kClRanks; ++p) s[r] += slots[p][r];
            }
            halpern_decide(c, s, A.chunk);
        }
        __syncthreads();
        if (c.done) break;
        if (c.restart_now) {
            for (int j = tid; j < cols; j += nt) x[j] = x0[j] = xf[c0 + j];
            for (int i = tid; i < rows; i += nt) y[i] = y0[i] = yf[r0 + i];
        } else {
            for (int i = tid; i < rows; i += nt) cl_put(yf, r0 + i, y[i], 0, 1);
        }
        cl_sync();
    }
    for (int j = tid; j < cols; j += nt) {
        A.x[c0 + j] = x[j];
        A.x0[c0 + j] = x0[j];
    }
    for (int i = tid; i < rows; i += nt) {
        A.y[r0 + i] = y[i];
        A.y0[r0 + i] = y0[i];
    }
    if (rank == 0 && tid == 0) *A.ctl = c;
}

} // namespace vk
