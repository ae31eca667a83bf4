// Scalar control of one cycle, shared by the control kernels and the
// resident-run kernels.  No product below feeds a sum, so contraction
// settings do not change the results.
#pragma once

#include "ensc_device.cuh"

namespace ensc {

// x / c for a divisor used many times, rc = 1 / c rounded to nearest: a
// quotient estimate corrected twice by its exact remainder, which rounds as the
// division does (P. Markstein, "Computation of elementary functions on the IBM
// RISC System/6000 processor", 1990: an estimate within one unit in the last
// place and one correction with a correctly rounded reciprocal suffice; the
// first correction brings the estimate there).  For |x| >= 2^-969, below which
// the remainder x - q c may underflow, with c, rc and the quotient normal; a
// smaller x is off by a few units in the last place at most, a zero of either
// sign gives +0, and a non-finite x a non-finite quotient.  Five dependent
// operations without the branch and the call of a general division.
__device__ __forceinline__ double div_by(double x, double c, double rc) {
    double q = x * rc;
    q = __fma_rn(__fma_rn(-q, c, x), rc, q);
    return __fma_rn(__fma_rn(-q, c, x), rc, q);
}

// True when the instance must not begin another cycle (a status was raised,
// the step end, the cycle budget or the pause time is reached).
__device__ __forceinline__ bool cycle_stops(const Ctl* ctl, int32_t status) {
    return status || !(ctl->time < ctl->step_end) || ctl->cycles_done >= ctl->cycles_target ||
           !(ctl->time < ctl->pause_time);
}

// First half of update_minVertex_perMaterial_and_dt for the next cycle
// (exDyna3D.cpp:663-686) and computeSate's clock advance (:775-780): rotate
// dt_i_1 <- dt_i and advance time, unless the total-time clamp (:682-685)
// could fire, which needs the cycle's minimum element edge first
// (begin_exact).  Caller has checked done / step end.
__device__ __forceinline__ void cycle_begin(Ctl* ctl) {
    ctl->dts_cur = bits_ord(ctl->dts_next);
    ctl->dts_next = kInfBits;
    ctl->len_min = kInfBits;
    const double dt_prev = ctl->dt_i;
    ctl->dt_prev = dt_prev;
    const double time = ctl->time;
    const double time_prev = time + dt_prev;
    // the new dt is factor * min(edge / c, dts_cur) <= factor * dts_cur
    const double bound = ctl->dts_cur * ctl->factor;
    const double rem = ctl->total_time - time_prev;
    const int exact = (rem > 0.0 && rem < bound) ? 1 : 0;
    ctl->need_exact = exact;
    ctl->dt_final = 0;
    if (!exact) {
        double dt_i_1 = dt_prev;
        if (time + dt_i_1 > ctl->step_end) {
            const double r = ctl->step_end - time;
            dt_i_1 = r;
            ctl->dt_i = r;
            ctl->dt_final = 1;
        }
        ctl->dt_i_1 = dt_i_1;
        double t = time + dt_i_1;
        if (t > ctl->total_time) t = ctl->total_time;
        ctl->time = t;
    }
}

// Rest of update_minVertex_perMaterial_and_dt and run()'s clamp for a cycle
// that needed the exact edge minimum (len_min_bits: that minimum, as
// ordered bits).
__device__ __forceinline__ void begin_exact(Ctl* ctl, unsigned long long len_min_bits) {
    const double time = ctl->time;
    double dt_i_1 = ctl->dt_prev;
    const double time_prev = time + dt_i_1;
    double d = bits_ord(len_min_bits) / ctl->wos;
    d = d < ctl->dts_cur ? d : ctl->dts_cur;
    double dt_i = d * ctl->factor;
    if ((ctl->total_time - time_prev) < dt_i && (ctl->total_time - time_prev) > 0.0) {
        dt_i = ctl->total_time - time_prev;
        dt_i_1 = dt_i;
    }
    if (time + dt_i_1 > ctl->step_end) {
        const double r = ctl->step_end - time;
        dt_i = r;
        dt_i_1 = r;
    }
    ctl->dt_i = dt_i;
    ctl->dt_i_1 = dt_i_1;
    ctl->dt_final = 1;
    double t = time + dt_i_1;
    if (t > ctl->total_time) t = ctl->total_time;
    ctl->time = t;
}

// The cycle's stable dt once the element pass has left its edge minimum
// (update_minVertex_perMaterial_and_dt, exDyna3D.cpp:673-679); inv_wos =
// 1 / ctl->wos.
__device__ __forceinline__ double cycle_dt(const Ctl* ctl, unsigned long long len_min_bits, double inv_wos) {
    if (ctl->dt_final) return ctl->dt_i;
    double d = div_by(bits_ord(len_min_bits), ctl->wos, inv_wos);
    const double tmp = ctl->dts_cur;
    d = d < tmp ? d : tmp;
    return d * ctl->factor;
}

// Minimum squared edge of a hexahedron from its corner coordinates
// (min_ele_edge, exDyna3D.cpp:1173-1220), as the element pass evaluates it.
__device__ __forceinline__ double min_edge_sq(const double (&xyz)[8][3]) {
    constexpr int A0[12] = {0, 1, 2, 3, 4, 5, 6, 7, 0, 1, 2, 3};
    constexpr int A1[12] = {1, 2, 3, 0, 5, 6, 7, 4, 4, 5, 6, 7};
    double m = 1.7976931348623157e308;
#pragma unroll
    for (int k = 0; k < 12; ++k) {
        const double dx = xyz[A1[k]][0] - xyz[A0[k]][0];
        const double dy = xyz[A1[k]][1] - xyz[A0[k]][1];
        const double dz = xyz[A1[k]][2] - xyz[A0[k]][2];
        const double t = __fma_rn(dz, dz, __fma_rn(dy, dy, dx * dx));
        m = t < m ? t : m;
    }
    return m;
}

}  // namespace ensc
