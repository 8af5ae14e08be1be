// pf_sym.cuh -- one element's product from its packed symmetric FP32 or FP16
// record by one warp: the bodies shared by the bulk-copy kernels
// (pf_elem_sym.cu, pf_elem_h16.cu) and the resident PCG (pf_resident.cu).
//
// Lane l < 30 owns rows and freedoms l and l+30 (node l/3 and node l/3+10,
// both in direction l%3).
#pragma once
#include "pf_device.cuh"
#include "pf_tc.cuh"

#include <cuda_fp16.h>

namespace pf {
namespace sym {

constexpr int kPSlot = 120;                    // floats of p per warp
constexpr int kWords32 = 1832, kWords16 = 916; // 4-byte words of a record
constexpr int kBytes32 = kWords32 * 4, kBytes16 = kWords16 * 4;

// p of an element, less its mean translation, into the warp's slot pp.  Lanes 30
// and 31 pass zeros.
// K_e t = 0 for a rigid translation t, so the subtraction changes nothing in
// exact arithmetic; in FP32 it keeps the translation of a smooth p out of
// the rounding of p, of storkm's entries and of the sums (errors that grow
// with the square of the mesh size on the lowest modes).  The mean is formed
// from the FP32 high parts -- any translation serves -- and (hi - t) + lo
// recovers p - t to FP32 accuracy relative to p - t.
//   FP32: p_e twice over, so that (i + s) mod 60 needs no wrap
//   FP16: pairs (p[i], p[i+30 mod 60]), one 8-byte load per step of the walk
template <bool H16>
__device__ __forceinline__ void put_p(int lane, double pa, double pb, float *pp)
{
    float ha, la, hb, lb;
    tc::split_f64(pa, ha, la);
    tc::split_f64(pb, hb, lb);
    const float t = 0.05f * tc::sum_mod3(ha + hb, lane);
    if (lane < 30) {
        const float qa = (ha - t) + la, qb = (hb - t) + lb;
        if constexpr (H16) {
            float2 *p2 = reinterpret_cast<float2 *>(pp);
            p2[lane] = make_float2(qa, qb);
            p2[lane + 30] = make_float2(qb, qa);
        } else {
            pp[lane] = qa;
            pp[lane + 60] = qa;
            pp[lane + 30] = qb;
            pp[lane + 90] = qb;
        }
    }
}

// Rows l and l+30 of P K_e times the projected p in pp (FP32 record D): four
// running sums over the diagonals.  Step d pairs forward distance d
// (K(l, l+d), K(l+30, l+30+d)) with backward distance 30-d (K(l+30, l+d),
// K(l, l+30+d)), which use the same two p values.  Every address is the lane
// plus a constant.
__device__ __forceinline__ void walk32(int lane, const float *D, const float *pp, float &acc_a, float &acc_b)
{
    acc_a = acc_b = 0.f;
    if (lane < 30) {
        const float *Dl = D + lane, *Dw = D + lane + 60;   // Dw: entries (l - t) mod 60 for t > l
        const float *pl = pp + lane;
        float f0 = Dl[0] * pl[0], f1 = Dl[30] * pl[30], g0 = 0.f, g1 = 0.f;
#pragma unroll
        for (int d = 1; d < 30; ++d) {
            const int t = 30 - d;
            const float p0 = pl[d], p1 = pl[30 + d];
            f0 = fmaf(Dl[60 * d], p0, f0);                              // K(l, l+d)
            f1 = fmaf(Dl[60 * d + 30], p1, f1);                         // K(l+30, l+30+d)
            g1 = fmaf(Dl[60 * t + d], p0, g1);                          // K(l+30, l+d) = D[t][l+d]
            g0 = fmaf((lane < t ? Dw : Dl)[59 * t], p1, g0);            // K(l, l-t) = D[t][(l-t) mod 60]
        }
        const float d30 = Dl[1800];                                     // K(l, l+30)
        f0 = fmaf(d30, pl[30], f0);
        f1 = fmaf(d30, pl[0], f1);
        acc_a = f0 + g0;
        acc_b = f1 + g1;
    }
}

// The same from an FP16 record (half2 words and the element's scale)
__device__ __forceinline__ void walk16(int lane, const uint32_t *Wd, const float *pp, float &acc_a, float &acc_b)
{
    acc_a = acc_b = 0.f;
    if (lane < 30) {
        const float2 *pl = reinterpret_cast<const float2 *>(pp) + lane;
        const float2 p00 = pl[0];   // (p[l], p[l+30])
        const float2 w0 = __half22float2(*reinterpret_cast<const __half2 *>(Wd + lane));
        float f0 = w0.x * p00.x, f1 = w0.y * p00.y, g0 = 0.f, g1 = 0.f;
#pragma unroll
        for (int d = 1; d < 30; ++d) {
            const int t = 30 - d;
            const float2 pd = pl[d];   // (p[l+d], p[l+d+30 mod 60])
            const float p0 = pd.x, p1 = pd.y;
            const float2 wf = __half22float2(*reinterpret_cast<const __half2 *>(Wd + 30 * d + lane));
            f0 = fmaf(wf.x, p0, f0);                                      // K(l, l+d)
            f1 = fmaf(wf.y, p1, f1);                                      // K(l+30, l+30+d)
            const bool wrap = lane >= t;                                  // l + d >= 30
            const float2 wb =
                __half22float2(*reinterpret_cast<const __half2 *>(Wd + 30 * t + (wrap ? lane - t : lane + d)));
            g1 = fmaf(wrap ? wb.y : wb.x, p0, g1);                        // K(l+30, l+d)
            g0 = fmaf(wrap ? wb.x : wb.y, p1, g0);                        // K(l, l+d+30)
        }
        const float d30 = __half2float(reinterpret_cast<const __half *>(Wd + 900)[lane]);   // K(l, l+30)
        f0 = fmaf(d30, p00.y, f0);
        f1 = fmaf(d30, p00.x, f1);
        const float sc = __uint_as_float(Wd[915]);
        acc_a = (f0 + g0) * sc;
        acc_b = (f1 + g1) * sc;
    }
}

// The projection of the result (t'K_e = 0 as well), so that the product
// stays symmetric: u_e = P K_e P p_e
__device__ __forceinline__ void project_result(int lane, float &acc_a, float &acc_b)
{
    const float t = 0.05f * tc::sum_mod3(acc_a + acc_b, lane);
    acc_a -= t;
    acc_b -= t;
}

}  // namespace sym
}  // namespace pf
