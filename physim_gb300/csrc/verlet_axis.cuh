// verlet_axis.cuh -- one coordinate's verlet update (integrators/src/verlet.rs:
// 24-82) in f64 in the reference's operation order.
#pragma once

namespace pg {

// verlet.rs:33-39 (initial, Taylor step) and verlet.rs:64-70 (regular).
__device__ __forceinline__ void verlet_axis(double &x, double &v, double &p, double a, double dt,
                                            double dt2, bool initial)
{
    double xn, vn;
    if (initial) {
        // x + vx*dt + 0.5*a*dt^2 ; vx + a*dt
        xn = __dadd_rn(__dadd_rn(x, __dmul_rn(v, dt)), __dmul_rn(__dmul_rn(0.5, a), dt2));
        vn = __dadd_rn(v, __dmul_rn(a, dt));
    } else {
        // 2*x - prev + a*dt^2 ; (x' - x)/dt
        xn = __dadd_rn(__dsub_rn(__dmul_rn(2.0, x), p), __dmul_rn(a, dt2));
        vn = __ddiv_rn(__dsub_rn(xn, x), dt);
    }
    p = x;
    x = xn;
    v = vn;
}

}  // namespace pg
