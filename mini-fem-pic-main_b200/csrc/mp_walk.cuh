// The reference's barycentric coordinates and tet walk in FP64, bit for bit
// (every operation rounded on its own, in the reference's order: no FMA).
// Shared by the push kernels and the adjoint.
#pragma once

#include "mp_internal.h"

namespace mp {

constexpr double ONE_SIXTH = 1.0 / 6.0;

// 32 bytes of a tet's record in one load (32-byte aligned, read-only).  A warp's
// lanes read up to 32 records, and a load costs the L1 a pass per record whatever
// its width: with 16-byte and scalar loads the mixed push kept the L1 at 74 % of
// its rate.  Push kernel in one wave of CTAs, before -> with these: mixed, 39M ions on
// the 32^3 box minus the sphere 1.23 -> 1.08 ms, 2M on the 20^3 box 55 -> 51 us; FP64, 2M
// 85 -> 80 us.  (The mixed push's neighbours and nodes are
// read when needed: loaded with the gradients they cost registers, 57 us at 2M.)
__device__ __forceinline__ void load32(const double *p, double (&v)[4]) {
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3]) : "l"(p));
}
__device__ __forceinline__ void load32(const float *p, float (&v)[8]) {
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
        : "l"(p));
}
__device__ __forceinline__ void load32(const int *p, int (&v)[8]) {
    asm("ld.global.nc.v8.s32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
        : "l"(p));
}

// Numerators q_i = (1.0/6.0)*(alpha_i - x*beta_i + y*gamma_i - z*delta_i) of
// the barycentric weights lambda_i = q_i/volume (src/meshes.h:84-85), in the
// reference's order, every operation rounded on its own.
__device__ __forceinline__ void numerators_fp64(const TetRec *__restrict__ t, double x, double y, double z,
                                                double q[4]) {
    double al[4], be[4], ga[4], de[4];
    load32(t->alpha, al);
    load32(t->beta, be);
    load32(t->gamma, ga);
    load32(t->delta, de);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        double w = __dsub_rn(al[i], __dmul_rn(x, be[i]));
        w = __dadd_rn(w, __dmul_rn(y, ga[i]));
        w = __dsub_rn(w, __dmul_rn(z, de[i]));
        q[i] = __dmul_rn(ONE_SIXTH, w);
    }
}

// The reference's lambda_i = q_i/volume, correctly rounded.
__device__ __forceinline__ void lambdas_fp64(const TetRec *__restrict__ t, double x, double y, double z,
                                             double lc[4]) {
    double q[4];
    numerators_fp64(t, x, y, z, q);
    const double vol = __ldg(&t->volume);
#pragma unroll
    for (int i = 0; i < 4; i++) lc[i] = __ddiv_rn(q[i], vol);
}

// XtoLtet (src/meshes.h:75-100) with a hop limit.  Returns 1 inside, 0 left the
// domain, -1 hop limit reached (cell is then the last tet visited).
//
// EXACT_CMP (every tet volume below 1): the inside test runs on the numerators,
// without the four divisions, and takes the same decisions.  With V > 0 and
// lambda = RN(q/V):
//   lambda < 0  <=>  q < 0   (q/V cannot round to -0 when V < 1: |q| >= 2^-1074)
//   lambda > 1  <=>  q > V   (if q > V then q >= V + ulp(V) > V(1 + 2^-53), the
//                             rounding midpoint above 1; if q <= V then q/V <= 1)
// and NaN compares false either way.  An inside particle's weights for the
// scatter are then q*RN(1/V) (within 2 ulp of lambda).  A particle outside its
// tet needs the exact lambdas for the hop (first minimum, strict <), so those
// are divided.  vol: the volume of the tet the walk starts in.
template <bool EXACT_CMP = false>
__device__ __forceinline__ int walk_fp64(const TetRec *__restrict__ tets, int &cell, double x, double y, double z,
                                         double vol, double lc[4], int limit, int &hops,
                                         int *exit_face = nullptr) {
    for (;;) {
        const TetRec *t = tets + cell;
        double q[4];
        numerators_fp64(t, x, y, z, q);
        if (EXACT_CMP) {
            bool inside = true;
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (q[i] < 0 || q[i] > vol) inside = false;
            if (inside) {
                const double rv = __drcp_rn(vol);
#pragma unroll
                for (int i = 0; i < 4; i++) lc[i] = __dmul_rn(q[i], rv);
                return 1;
            }
#pragma unroll
            for (int i = 0; i < 4; i++) lc[i] = __ddiv_rn(q[i], vol);
        } else {
            bool inside = true;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                lc[i] = __ddiv_rn(q[i], vol);
                if (lc[i] < 0 || lc[i] > 1.0) inside = false;
            }
            if (inside) return 1;
        }
        int min_i = 0;
        double min_lc = lc[0];
#pragma unroll
        for (int i = 1; i < 4; i++)
            if (lc[i] < min_lc) {
                min_lc = lc[i];
                min_i = i;
            }
        int nb = __ldg(&t->cell_con[min_i]);
        if (nb < 0) {
            if (exit_face) *exit_face = min_i;  // the face opposite vertex min_i of `cell`
            return 0;
        }
        if (hops >= limit) return -1;
        cell = nb;
        vol = __ldg(&tets[nb].volume);
        hops++;
    }
}

}  // namespace mp
