// stage_dmma_columns.cuh -- column phase of an element of 8 points per direction on the FP64
// tensor cores, one warp of four per residual role (stage_dmma.cuh has the reasons and the
// rest of the tile; the FP64 elements of the FP32-bulk class use it too).
// Fragment layout (m8n8k4, A row-major 8x4, B column-major 4x8, C 8x8): lane
// L = 4g + t holds A[g][t], B[t][g], C[g][2t] and C[g][2t+1].
#pragma once
#include "stage_mma.cuh"

namespace nwb {
namespace stage {

// Column phase of one warp: field src -> dst, residual components ROLE (0: x, 1: y) on all
// planes and z on planes 4 ROLE .. 4 ROLE + 3.  CS: component stride of the shared tile (even).
// zlo, zhi: the lifted flux of component ROLE on the faces across t at the lane's nodes.
template <int ROLE, int CS>
__device__ __forceinline__ void dmma8_columns(const StageParams& P, const double* su, const double* V,
                                              const double* Fl, int g, int t, int dst, double d0, double d1,
                                              double rx, double sy, double tz, long long ebase,
                                              const double* __restrict__ Dc, const double2* zlo,
                                              const double2* zhi) {
    const double A = P.a, B = P.b, DT = P.dt;
    const bool kread = (P.kio & kKRead) != 0, kwrite = (P.kio & kKWrite) != 0;
    const int hf = dst == 0 ? 0 : 1;
    const long long S = P.stride;
    const int m0 = 8 * g + 2 * t;  // the lane's first node in a plane
    // its two node columns of the component differentiated along t
    double2 col[8];
#pragma unroll
    for (int l = 0; l < 8; ++l) col[l] = *reinterpret_cast<const double2*>(V + (1 - ROLE) * CS + 64 * l + m0);
    double* const k1 = P.k + (dst + ROLE) * S + ebase + m0;
    double* const k2 = P.k + (dst + 2) * S + ebase + m0;
    double* const o1 = P.u_out + (dst + ROLE) * S + ebase + m0;
    double* const o2 = P.u_out + (dst + 2) * S + ebase + m0;
    auto load_k = [&](const double* p) {
        return kread ? ld_state(reinterpret_cast<const double2*>(p)) : make_double2(0.0, 0.0);
    };
    auto update = [&](double* kp, double* op, const double* up, double2 kold, double r0, double r1) {
        const double kn0 = A * kold.x + DT * r0, kn1 = A * kold.y + DT * r1;
        const double2 uo = *reinterpret_cast<const double2*>(up);
        if (kwrite) __stcs(reinterpret_cast<double2*>(kp), make_double2(kn0, kn1));
        __stcs(reinterpret_cast<double2*>(op), make_double2(uo.x + B * kn0, uo.y + B * kn1));
    };
    const bool onx = t == 0 || t == 3, ony = g == 0 || g == 7;
    const double* Fx = Fl + ((t == 0 ? 3 : 1) * 4 + 2 * hf) * 64 + g;      // x faces: y, z components
    const double* Fy = Fl + ((g == 0 ? 0 : 2) * 4 + 2 * hf) * 64 + 2 * t;  // y faces: z, x components
    double2 n1 = load_k(k1), n2 = make_double2(0.0, 0.0);
    if (ROLE == 0) n2 = load_k(k2);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const bool z_now = (k >= 4) == (ROLE == 1), z_next = (k + 1 >= 4) == (ROLE == 1);
        const double2 c1 = n1, c2 = n2;
        if (k < 7) {
            n1 = load_k(k1 + 64 * (k + 1));
            if (z_next) n2 = load_k(k2 + 64 * (k + 1));
        }
        const double* Vz = V + 2 * CS + 64 * k;
        double a0 = 0.0, a1 = 0.0;
        if constexpr (ROLE == 0) {  // s (swapped form): B[t][g] = V(i = g, l = t, k)
            dmma_f64(a0, a1, d0, Vz[8 * t + g]);
            dmma_f64(a0, a1, d1, Vz[8 * (4 + t) + g]);
        } else {  // r (original form): A[g][t] = V(l = t, j = g, k)
            dmma_f64(a0, a1, Vz[8 * g + t], d0);
            dmma_f64(a0, a1, Vz[8 * g + 4 + t], d1);
        }
        // t: sums over the cached columns, D(k, l) from Dc (the parameter bank when the
        // caller has it there, else shared memory: the same values either way)
        double b0 = 0.0, b1 = 0.0;
#pragma unroll
        for (int l = 0; l < 8; ++l) {
            const double dk = Dc[k + 8 * l];
            b0 += dk * col[l].x;
            b1 += dk * col[l].y;
        }
        double r0, r1;
        if constexpr (ROLE == 0) {
            r0 = sy * a0 - tz * b0;
            r1 = sy * a1 - tz * b1;
            if (ony) {
                const double2 y = *reinterpret_cast<const double2*>(Fy + 64 + 8 * k);
                r0 += y.x;
                r1 += y.y;
            }
        } else {
            r0 = tz * b0 - rx * a0;
            r1 = tz * b1 - rx * a1;
            if (onx) {
                const double x = Fx[8 * k];
                if (t == 0) r0 += x;
                else r1 += x;
            }
        }
        if (k == 0 || k == 7) {
            const double2 z = k == 0 ? *zlo : *zhi;
            r0 += z.x;
            r1 += z.y;
        }
        if (z_now) {
            const double* Vy = V + CS + 64 * k;
            const double* Vx = V + 64 * k;
            double yr0 = 0.0, yr1 = 0.0, xs0 = 0.0, xs1 = 0.0;
            dmma_f64(yr0, yr1, Vy[8 * g + t], d0);
            dmma_f64(yr0, yr1, Vy[8 * g + 4 + t], d1);
            dmma_f64(xs0, xs1, d0, Vx[8 * t + g]);
            dmma_f64(xs0, xs1, d1, Vx[8 * (4 + t) + g]);
            double q0 = rx * yr0 - sy * xs0, q1 = rx * yr1 - sy * xs1;
            // face order: y-, x+, y+, x- (add_lifts_xy)
            double x = 0.0;
            double2 y = make_double2(0.0, 0.0);
            if (onx) x = Fx[64 + 8 * k];
            if (ony) y = *reinterpret_cast<const double2*>(Fy + 8 * k);
            const bool xfirst = t == 3 && g == 7;
            q0 = (q0 + y.x) + (t == 0 ? x : 0.0);
            const double xb = t == 3 ? x : 0.0;
            q1 = (q1 + (xfirst ? xb : y.y)) + (xfirst ? y.y : xb);
            update(k2 + 64 * k, o2 + 64 * k, su + (dst + 2) * CS + 64 * k + m0, c2, q0, q1);
        }
        // LSRK45 (src/device/dg_kernels.cu:404-406), FP64
        update(k1 + 64 * k, o1 + 64 * k, su + (dst + ROLE) * CS + 64 * k + m0, c1, r0, r1);
    }
}

}  // namespace stage
}  // namespace nwb
