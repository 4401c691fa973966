// The restarted Halpern scheme on a resident model (vk_resident.cuh): the
// iterations, checks and restarts of vk_halpern.cu, `chunks` check intervals in
// one launch.
#pragma once

#include "vk_halpern_ctl.cuh"
#include "vk_resident.cuh"

namespace vk {

template <class T>
struct RsHalArgs {
    const int *ro_a, *ci_a, *ro_t, *ci_t, *ro_q, *ci_q;
    const T *va, *vt, *vq;
    const int *part_a, *part_t; // row and column boundaries of the CTAs
    int cap_a, cap_t, cap_q, rows, cols; // the largest shares: nonzeros, rows, columns
    T *x, *x0, *xbar, *xhat, *y, *y0, *yhat;
    const T *c, *l, *u, *cs, *rl, *ru, *rs;
    HalCtl *ctl;
    double *partials;
    unsigned *counter;
    int *err;
    int chunk, chunks;
};

// Byte offsets in a CTA's dynamic shared memory.
template <class T, class I>
struct RsHalLayout {
    size_t va, vt, vq, ia, it, iq, roa, rot, roq, prod, xs, ys, bytes;
    static constexpr int kXs = 5, kYs = 4; // own columns: x, x0, c, l, u (QP: qx, qh too); own rows: y, y0, rl, ru
    __host__ __device__ RsHalLayout(int cap_a, int cap_t, int cap_q, int rows, int cols, bool qp) {
        size_t o = 0;
        const auto take = [&](size_t b) {
            const size_t at = o;
            o = (o + b + 15) & ~static_cast<size_t>(15);
            return at;
        };
        const size_t a = cap_a, t = cap_t, q = cap_q;
        va = take(sizeof(T) * a);
        vt = take(sizeof(T) * t);
        vq = take(sizeof(T) * q);
        ia = take(sizeof(I) * a);
        it = take(sizeof(I) * t);
        iq = take(sizeof(I) * q);
        roa = take(4 * (static_cast<size_t>(rows) + 1));
        rot = take(4 * (static_cast<size_t>(cols) + 1));
        roq = take(qp ? 4 * (static_cast<size_t>(cols) + 1) : 0);
        prod = take(sizeof(double) * (a > t ? (a > q ? a : q) : (t > q ? t : q))); // the checks' are float64
        xs = take(sizeof(T) * (kXs + (qp ? 2 : 0)) * static_cast<size_t>(cols));
        ys = take(sizeof(T) * kYs * static_cast<size_t>(rows));
        bytes = o;
    }
};

template <class T, class I, bool QP>
__global__ void __launch_bounds__(kRsThreads, 1) rs_halpern_kernel(RsHalArgs<T> A) {
    constexpr int kTab = 64; // lambda of the next iterations
    extern __shared__ __align__(16) unsigned char rs_smem[];
    __shared__ HalCtl c;
    __shared__ double scratch[32 * kCheckSums], totals[kCheckSums];
    __shared__ T lams[kTab];
    if (A.ctl->done) return; // the same for the whole grid
    const int tid = threadIdx.x, nt = blockDim.x;
    const int r0 = A.part_a[blockIdx.x], rows = A.part_a[blockIdx.x + 1] - r0;
    const int c0 = A.part_t[blockIdx.x], cols = A.part_t[blockIdx.x + 1] - c0;
    const RsHalLayout<T, I> lay(A.cap_a, A.cap_t, A.cap_q, A.rows, A.cols, QP);
    const auto vec = [&](size_t o) { return reinterpret_cast<T *>(rs_smem + o); };
    const auto ind = [&](size_t o) { return reinterpret_cast<I *>(rs_smem + o); };
    const auto off = [&](size_t o) { return reinterpret_cast<int *>(rs_smem + o); };
    T *prod = vec(lay.prod);
    double *prod64 = reinterpret_cast<double *>(rs_smem + lay.prod);
    T *x = vec(lay.xs), *x0 = x + A.cols, *cc = x0 + A.cols, *l = cc + A.cols, *u = l + A.cols;
    T *qx = u + A.cols, *qh = qx + A.cols; // QP only: Q^ x and, in a check, Q^ x^
    T *y = vec(lay.ys), *y0 = y + A.rows, *rl = y0 + A.rows, *ru = rl + A.rows;
    RsBarrier bar{A.counter, A.err};
    if (tid == 0) c = *A.ctl;
    const auto sa = rs_load<T, I>(A.ro_a, A.ci_a, A.va, r0, r0 + rows, vec(lay.va), ind(lay.ia), off(lay.roa));
    const auto st = rs_load<T, I>(A.ro_t, A.ci_t, A.vt, c0, c0 + cols, vec(lay.vt), ind(lay.it), off(lay.rot));
    RsSide<T, I> sq{};
    if (QP) sq = rs_load<T, I>(A.ro_q, A.ci_q, A.vq, c0, c0 + cols, vec(lay.vq), ind(lay.iq), off(lay.roq));
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
    __syncthreads();
    // qx = Q^ x over the own columns (QP)
    const auto q_pass = [&] {
        rs_products(sq, A.x, prod);
        rs_rows(sq, prod, [&](int j, T sum) { qx[j] = sum; });
        __syncthreads();
    };
    if (QP) {
        q_pass();
        if (!bar.sync()) return; // x is read everywhere before anyone writes it
    }

    struct ColIn {
        T x, x0, c, l, u;
    };
    struct RowIn {
        T y, y0, lo, hi;
    };
    for (int ch = 0; ch < A.chunks; ++ch) {
        const T tau = static_cast<T>(c.tau), sigma = static_cast<T>(c.sigma), rho = static_cast<T>(c.rho);
        const double kb = static_cast<double>(c.k_base);
        double dx2 = 0.0, dx0 = 0.0, dy2 = 0.0, dy0 = 0.0; // of the check's iteration
        for (int it = 0; it < A.chunk; ++it) {
            if (it % kTab == 0) {
                __syncthreads();
                if (tid < kTab) lams[tid] = static_cast<T>((kb + it + tid + 1.0) / (kb + it + tid + 2.0));
                __syncthreads();
            }
            const T lam = lams[it % kTab];
            const bool check = it == A.chunk - 1;
            rs_products(st, A.y, prod);
            const auto column = [&](int j) { return ColIn{x[j], x0[j], QP ? cc[j] + qx[j] : cc[j], l[j], u[j]}; };
            rs_rows(st, prod, column, [&](int j, T sum, const ColIn &p) {
                const T xv = p.x, xz = p.x0;
                const T xh = clampbox(xv - tau * (p.c + sum), p.l, p.u);
                A.xbar[c0 + j] = T(2) * xh - xv;
                const T xn = lam * ((T(1) + rho) * xh - rho * xv) + (T(1) - lam) * xz;
                x[j] = xn;
                if (QP) A.x[c0 + j] = xn;
                if (check) {
                    A.xhat[c0 + j] = xh;
                    const double d0 = static_cast<double>(xh) - static_cast<double>(xv);
                    const double d1 = static_cast<double>(xh) - static_cast<double>(xz);
                    dx2 += d0 * d0;
                    dx0 += d1 * d1;
                }
            });
            if (!bar.sync()) return;
            rs_products(sa, A.xbar, prod);
            const auto dual = [&](int i) { return RowIn{y[i], y0[i], sigma * rl[i], sigma * ru[i]}; };
            rs_rows(sa, prod, dual, [&](int i, T sum, const RowIn &p) {
                const T yv = p.y, yz = p.y0;
                const T v = yv + sigma * sum;
                const T yh = v - clampbox(v, p.lo, p.hi);
                const T yn = lam * ((T(1) + rho) * yh - rho * yv) + (T(1) - lam) * yz;
                A.y[r0 + i] = yn;
                y[i] = yn;
                if (check) {
                    A.yhat[r0 + i] = yh;
                    const double d0 = static_cast<double>(yh) - static_cast<double>(yv);
                    const double d1 = static_cast<double>(yh) - static_cast<double>(yz);
                    dy2 += d0 * d0;
                    dy0 += d1 * d1;
                }
            });
            if (QP) { // the next column pass's Q^ x
                __syncthreads();
                q_pass();
            }
            if (!bar.sync()) return;
        }
        // the check: K x^, (Q^ x^,) K'y^
        double s[kCheckSums] = {dx2, dx0, dy2, dy0};
        rs_products(sa, A.xhat, prod64);
        rs_rows(sa, prod64, [&](int i, double sum) {
            kkt_row_terms(sum, rl[i], ru[i], A.rs[r0 + i], A.yhat[r0 + i], s + kColCheckSums + kRowCheckSums);
        });
        __syncthreads();
        if (QP) {
            rs_products(sq, A.xhat, prod64);
            rs_rows(sq, prod64, [&](int j, double sum) { qh[j] = static_cast<T>(sum); });
            __syncthreads();
        }
        rs_products(st, A.yhat, prod64);
        rs_rows(st, prod64, [&](int j, double sum) {
            kkt_col_terms(sum, cc[j], QP ? static_cast<double>(qh[j]) : 0.0, A.cs[c0 + j], l[j], u[j], A.xhat[c0 + j],
                          s + kCheckSums - kKktColSums);
        });
        if (!rs_sum<kCheckSums>(s, A.partials, scratch, totals, bar)) return;
        if (tid == 0) halpern_decide(c, totals, A.chunk); // the same numbers, the same decision in every CTA
        __syncthreads();
        if (c.done) break;
        if (c.restart_now) {
            for (int j = tid; j < cols; j += nt) {
                x[j] = x0[j] = A.xhat[c0 + j];
                if (QP) {
                    A.x[c0 + j] = x[j];
                    qx[j] = qh[j];
                }
            }
            for (int i = tid; i < rows; i += nt) y[i] = y0[i] = A.y[r0 + i] = A.yhat[r0 + i];
            if (!bar.sync()) return;
        }
    }
    for (int j = tid; j < cols; j += nt) {
        A.x[c0 + j] = x[j];
        A.x0[c0 + j] = x0[j];
    }
    for (int i = tid; i < rows; i += nt) A.y0[r0 + i] = y0[i];
    if (blockIdx.x == 0 && tid == 0) *A.ctl = c;
}

} // namespace vk
