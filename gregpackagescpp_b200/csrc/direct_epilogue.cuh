// The integrators' updates, applied by whichever kernel finishes a body's force sum.
#pragma once

#include "gtd_internal.cuh"

namespace gtd {

// The method's update of body i from its summed force (ax, ay, az), in FP64.
__device__ __forceinline__ void apply_epilogue(const StepArgs &st, int epi, int64_t i, double ax, double ay, double az) {
    const double h = st.h, h2 = 0.5 * st.h;
    if (epi == EPI_ACC) {  // the force alone: position and velocity are not read
        st.acc[i] = make_double4(ax, ay, az, 0.0);
        return;
    }
    if (epi == EPI_ACC3) {
        double *o = reinterpret_cast<double *>(st.acc) + 3 * i;
        o[0] = ax;
        o[1] = ay;
        o[2] = az;
        return;
    }
    const double4 x = st.cur[i];
    double4 v = st.vel[i];
    switch (epi) {
        case EPI_KDK: {
            st.acc[i] = make_double4(ax, ay, az, 0.0);
            v.x = fma(h2, ax, v.x); v.y = fma(h2, ay, v.y); v.z = fma(h2, az, v.z);
            if (!st.last) {
                v.x = fma(h2, ax, v.x); v.y = fma(h2, ay, v.y); v.z = fma(h2, az, v.z);
                st.dst[i] = make_double4(fma(h, v.x, x.x), fma(h, v.y, x.y), fma(h, v.z, x.z), x.w);
            }
            st.vel[i] = v;
            break;
        }
        case EPI_DKD: {
            st.acc[i] = make_double4(ax, ay, az, 0.0);
            v.x = fma(h, ax, v.x); v.y = fma(h, ay, v.y); v.z = fma(h, az, v.z);
            double4 y = make_double4(fma(h2, v.x, x.x), fma(h2, v.y, x.y), fma(h2, v.z, x.z), x.w);
            if (!st.last) y = make_double4(fma(h2, v.x, y.x), fma(h2, v.y, y.y), fma(h2, v.z, y.z), x.w);
            st.dst[i] = y;
            st.vel[i] = v;
            break;
        }
        case EPI_EULER: {
            st.acc[i] = make_double4(ax, ay, az, 0.0);
            st.dst[i] = make_double4(fma(h, v.x, x.x), fma(h, v.y, x.y), fma(h, v.z, x.z), x.w);
            v.x = fma(h, ax, v.x); v.y = fma(h, ay, v.y); v.z = fma(h, az, v.z);
            st.vel[i] = v;
            break;
        }
        case EPI_PREDICT: {
            const double hp = st.hp;
            st.acc[i] = make_double4(ax, ay, az, 0.0);
            st.pred_pos[i] = make_double4(fma(hp, v.x, x.x), fma(hp, v.y, x.y), fma(hp, v.z, x.z), x.w);
            st.pred_vel[i] = make_double4(fma(hp, ax, v.x), fma(hp, ay, v.y), fma(hp, az, v.z), 0.0);
            break;
        }
        case EPI_CORR_MEULER: {
            const double4 pv = st.pred_vel[i], a0 = st.acc[i];
            st.dst[i] = make_double4(fma(h2, v.x + pv.x, x.x), fma(h2, v.y + pv.y, x.y), fma(h2, v.z + pv.z, x.z),
                                     x.w);
            v.x = fma(h2, a0.x + ax, v.x); v.y = fma(h2, a0.y + ay, v.y); v.z = fma(h2, a0.z + az, v.z);
            st.vel[i] = v;
            break;
        }
        case EPI_CORR_MIDPOINT: {
            const double4 pv = st.pred_vel[i];
            st.dst[i] = make_double4(fma(h, pv.x, x.x), fma(h, pv.y, x.y), fma(h, pv.z, x.z), x.w);
            v.x = fma(h, ax, v.x); v.y = fma(h, ay, v.y); v.z = fma(h, az, v.z);
            st.vel[i] = v;
            break;
        }
        case EPI_KICK_DRIFT: {
            const double c = st.hp;
            v.x = fma(c, ax, v.x); v.y = fma(c, ay, v.y); v.z = fma(c, az, v.z);
            st.vel[i] = v;
            if (!st.last) st.dst[i] = make_double4(fma(h, v.x, x.x), fma(h, v.y, x.y), fma(h, v.z, x.z), x.w);
            break;
        }
        default:
            break;
    }
}

}  // namespace gtd
