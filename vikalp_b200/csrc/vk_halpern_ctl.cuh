// Control of the restarted reflected-Halpern scheme, shared by the kernels that
// run it: the control block, the step sizes, the terms of the relative KKT
// error and the stop / restart / primal-weight decision of a check.
#pragma once

#include "vk_common.cuh"
#include "vikalp_b200.h"

namespace vk {

constexpr int kColCheckSums = 2;       // |x^-x|^2, |x^-x0|^2
constexpr int kRowCheckSums = 2;       // |y^-y|^2, |y^-y0|^2
constexpr int kKktRowSums = 3;         // primal res^2, dual-obj rows, row-dual violations^2
constexpr int kKktColSums = 5;         // dual res^2, dual-obj cols, primal obj, box violation^2, x'Qx
constexpr int kCheckSums = kColCheckSums + kRowCheckSums + kKktRowSums + kKktColSums; // in this order

struct HalCtl {
    double eta, omega, tau, sigma;
    double r_restart, r_prev;
    double rel_p, rel_d, rel_gap, kkt;
    double bnorm, cnorm, offset, tol;
    double knorm, lq, rho, pad_d; // sigma_max(K), lambda_max(Q^) (0: LP), reflection
    double theta, freeze;                   // primal-weight smoothing; no update below this KKT
    double beta_suff, beta_nec, beta_art;   // restart thresholds
    long long k_base, total, limit, restarts, checks;
    int done, status, restart_now, pad;
};

// Step sizes for primal weight omega: tau = eta/omega, sigma = eta*omega.
// LP (lq == 0): eta = 0.99/|K| and full reflection rho = 1. QP: the explicit
// gradient step on 0.5 x'Q^x needs 1/tau - sigma |K|^2 >= L; eta solves
// tau L + eta^2 |K|^2 = 0.99^2 and the reflection is cut to
// rho = 0.99 (1 - 1/(2 kappa)), kappa = (1/tau - sigma |K|^2) / L, which keeps
// (1+rho) T - rho I nonexpansive (Condat's bound on the relaxation of the
// primal-dual iteration with a smooth term).
__host__ __device__ inline void step_params(double knorm, double lq, double omega, double &eta, double &rho) {
    if (!(lq > 0.0)) {
        eta = knorm > 0.0 ? 0.99 / knorm : 1.0;
        rho = 1.0;
        return;
    }
    const double k2 = knorm * knorm, b = lq / omega, c = 0.9801;
    eta = 2.0 * c / (b + sqrt(b * b + 4.0 * k2 * c));
    const double tau = eta / omega;
    const double kappa = (1.0 - eta * eta * k2) / (tau * lq);
    rho = fmin(1.0, 0.99 * (1.0 - 1.0 / (2.0 * kappa)));
}

// Relative-KKT terms of one row: a = (K x^)_i, scaled bounds, row scale r, y^_i.
__device__ __forceinline__ void kkt_row_terms(double a, double lo, double hi, double r, double y, double *red) {
    const double pr = (a - clampbox(a, lo, hi)) / r;
    red[0] += pr * pr;
    const double yl = smax(0.0, -y), yu = smax(0.0, y);
    if (yl > 0.0) {
        if (isfinite(lo)) red[1] += lo * yl; else red[2] += (r * yl) * (r * yl);
    }
    if (yu > 0.0) {
        if (isfinite(hi)) red[1] -= hi * yu; else red[2] += (r * yu) * (r * yu);
    }
}

// One column: kty = (K'y^)_j, q = (Q^ x^)_j (0 for an LP), column scale d.
__device__ __forceinline__ void kkt_col_terms(double kty, double c, double q, double d, double lo, double hi, double x,
                                              double *red) {
    const double lam = c + q + kty;
    const double vl = smax(0.0, lam), vu = smax(0.0, -lam);
    if (vl > 0.0) {
        if (isfinite(lo)) red[1] += lo * vl; else red[0] += (vl / d) * (vl / d);
    }
    if (vu > 0.0) {
        if (isfinite(hi)) red[1] -= hi * vu; else red[0] += (vu / d) * (vu / d);
    }
    red[2] += c * x;
    const double bx = (x - clampbox(x, lo, hi)) * d;
    red[3] += bx * bx;
    red[4] += x * q;
}

// One check: the sums of kCheckSums, then stop, restart and primal weight.
__device__ inline void halpern_decide(HalCtl &c, const double *s, int chunk) {
    const double dx2 = s[0], dx0 = s[1], dy2 = s[2], dy0 = s[3];
    const double rp2 = s[4], dobj_r = s[5], viol2 = s[6];
    const double rd2 = s[7], dobj_c = s[8], box2 = s[10], quad = s[11];
    const double pobj = s[9] + 0.5 * quad + c.offset;
    const double dobj = dobj_r + dobj_c - 0.5 * quad + c.offset;
    c.total += chunk;
    c.checks += 1;
    c.rel_p = (sqrt(rp2) + sqrt(box2)) / (1.0 + c.bnorm);
    c.rel_d = sqrt(rd2 + viol2) / (1.0 + c.cnorm);
    c.rel_gap = fabs(pobj - dobj) / (1.0 + fabs(pobj) + fabs(dobj));
    c.kkt = smax(smax(c.rel_p, c.rel_d), c.rel_gap);
    c.restart_now = 0;
    if (!(c.kkt == c.kkt)) { // NaN: stop, the host reports a numerical failure
        c.done = 1;
        c.status = VK_STATUS_NUMERICAL_FAILURE;
    } else if (c.kkt <= c.tol) {
        c.done = 1;
        c.status = VK_STATUS_OPTIMAL;
    } else if (c.total >= c.limit) {
        c.done = 1;
        c.status = VK_STATUS_ITERATION_LIMIT;
    } else {
        const double r = sqrt(c.omega * dx2 + dy2 / c.omega);
        const long long k = c.k_base + chunk;
        bool restart = false;
        if (c.r_restart < 0.0) {
            c.r_restart = r;
        } else {
            restart = (r <= c.beta_suff * c.r_restart) || (r <= c.beta_nec * c.r_restart && r > c.r_prev) ||
                      (static_cast<double>(k) >= c.beta_art * static_cast<double>(c.total));
        }
        c.r_prev = r;
        if (restart) {
            const double mx = sqrt(dx0), my = sqrt(dy0);
            if (mx > 1e-10 && my > 1e-10 && c.theta > 0.0 && c.kkt >= c.freeze)
                c.omega = exp(c.theta * log(my / mx) + (1.0 - c.theta) * log(c.omega));
            step_params(c.knorm, c.lq, c.omega, c.eta, c.rho);
            c.tau = c.eta / c.omega;
            c.sigma = c.eta * c.omega;
            c.k_base = 0;
            c.restarts += 1;
            c.restart_now = 1;
            c.r_restart = r;
        } else {
            c.k_base = k;
        }
    }
}

} // namespace vk
