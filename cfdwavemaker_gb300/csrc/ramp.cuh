// Ramp::ramp (Utils.cpp:42-68): the minimum of up to six clamped linear
// ramps in t, x and y, shared by the finishing pass of the API rows and the
// kernels that write the API rows themselves (regular waves; the irregular
// sums' combining pass).
#pragma once

namespace cfdwm {

struct RampDev {
    int init, flags;
    double lim[12];
};

__device__ __forceinline__ double d_ramp(const RampDev &r, double t, double x, double y) {
    if (!r.init) return 1.0;
    double v[6] = {t, t, x, x, y, y};
    double m = 1.0;
    for (int q = 0; q < 6; q++) {
        double rq = 1.0;
        if (r.flags & (1 << q)) {
            double a = (v[q] - r.lim[2 * q]) / (r.lim[2 * q + 1] - r.lim[2 * q]);
            rq = (q & 1) ? fmax(fmin(1. - a, 1.), 0.) : fmax(fmin(a, 1.), 0.);
        }
        m = (q == 0) ? rq : fmin(m, rq);
    }
    return m;
}

// The API rows written by the kernel that ends the evaluation: row[q][n], q =
// wave_SurfElev .. wave_nhPres (null: not wanted), and/or wave_Kinematics
// records [n][4], the ramp at (x, y, t) applied where one is set,
// p_nh = dp - rho g eta.  The rows are the caller's own arrays where they can
// be (run_batch), so a value is written once: through a scratch block of six
// rows and a copy per wanted row, a velocity call of a regular wave moved
// 128 B a point for its 56.
struct ApiRows {
    RampDev ramp;
    double rho, g;
    const double *x, *y, *t;
    double *row[6];
    double *kin;
    __host__ __device__ bool any() const {
        return row[0] || row[1] || row[2] || row[3] || row[4] || row[5] || kin;
    }
};

// The rows of point p, v[q] ramped where a ramp is set.
__device__ __forceinline__ void api_store(const ApiRows &a, long p, double v[6]) {
    if (a.ramp.init) {
        const double rr = d_ramp(a.ramp, a.t[p], a.x[p], a.y[p]);
        for (int q = 0; q < 6; q++) v[q] *= rr;
    }
#pragma unroll
    for (int q = 0; q < 6; q++)
        if (a.row[q]) a.row[q][p] = v[q];
    if (a.kin)
#pragma unroll
        for (int q = 0; q < 4; q++) a.kin[4 * p + q] = v[q];
}

}  // namespace cfdwm
