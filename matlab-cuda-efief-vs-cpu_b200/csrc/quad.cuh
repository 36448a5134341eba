// Device pieces of the quadrature shared by the assembly's kernels (assemble.cu,
// series.cu).
#pragma once

#include <cuda_runtime.h>

constexpr double kPi = 3.141592653589793238462643383279502884;

// I0 = int_T 1/R dS', J = int_T (r' - r)/R dS' for triangle (a0, a1, a2).
static __device__ void potential_integrals(const double3 a0, const double3 a1, const double3 a2, const double3 r,
                                    double &I0, double3 &J) {
    const double3 A[3] = {a0, a1, a2};
    double3 n = make_double3((a1.y - a0.y) * (a2.z - a0.z) - (a1.z - a0.z) * (a2.y - a0.y),
                             (a1.z - a0.z) * (a2.x - a0.x) - (a1.x - a0.x) * (a2.z - a0.z),
                             (a1.x - a0.x) * (a2.y - a0.y) - (a1.y - a0.y) * (a2.x - a0.x));
    const double nn = sqrt(n.x * n.x + n.y * n.y + n.z * n.z);
    n.x /= nn; n.y /= nn; n.z /= nn;
    const double d = n.x * (r.x - a0.x) + n.y * (r.y - a0.y) + n.z * (r.z - a0.z);
    const double ad = fabs(d);
    const double3 rho = make_double3(r.x - d * n.x, r.y - d * n.y, r.z - d * n.z);
    double s0 = 0.0, vx = 0.0, vy = 0.0, vz = 0.0;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const double3 p = A[i], q = A[(i + 1) % 3];
        double3 l = make_double3(q.x - p.x, q.y - p.y, q.z - p.z);
        const double ll = sqrt(l.x * l.x + l.y * l.y + l.z * l.z);
        l.x /= ll; l.y /= ll; l.z /= ll;
        const double3 u = make_double3(l.y * n.z - l.z * n.y, l.z * n.x - l.x * n.z, l.x * n.y - l.y * n.x);
        const double P0 = (p.x - rho.x) * u.x + (p.y - rho.y) * u.y + (p.z - rho.z) * u.z;
        const double lp = (q.x - rho.x) * l.x + (q.y - rho.y) * l.y + (q.z - rho.z) * l.z;
        const double lm = (p.x - rho.x) * l.x + (p.y - rho.y) * l.y + (p.z - rho.z) * l.z;
        const double R02 = P0 * P0 + d * d;
        const double Rp = sqrt(R02 + lp * lp), Rm = sqrt(R02 + lm * lm);
        double f;
        if (R02 < 1e-30 * (lp * lp + lm * lm)) {
            f = 0.0;   // point on the edge line: the terms vanish
        } else {
            // f = log((Rp + lp)/(Rm + lm)); R + l = R02/(R - l) where l < 0 avoids the cancellation
            const double np_ = lp >= 0.0 ? Rp + lp : R02 / (Rp - lp);
            const double nm_ = lm >= 0.0 ? Rm + lm : R02 / (Rm - lm);
            f = log(np_ / nm_);
        }
        double beta = 0.0;
        if (ad > 0.0) beta = atan(P0 * lp / (R02 + ad * Rp)) - atan(P0 * lm / (R02 + ad * Rm));
        s0 += P0 * f - ad * beta;
        const double t = 0.5 * (R02 * f + lp * Rp - lm * Rm);
        vx += u.x * t; vy += u.y * t; vz += u.z * t;
    }
    I0 = s0;
    J = make_double3(vx - d * n.x * s0, vy - d * n.y * s0, vz - d * n.z * s0);
}
