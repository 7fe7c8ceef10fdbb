// Winner-take-all of one pixel over a 16-byte aligned row of final sums (the byte form of the last SGM sweep).
#pragma once

#include <type_traits>

#include "common.cuh"
#include "kernels.h"

namespace apgcu {

// Where the winner-take-all writes, and its sub-pixel step.
struct WtaOut {
    float* disp;
    float* best;
    float* second;
    int subpixel;
    int sp_method;
    float sp_param;
    apg_subpixel_telemetry_t* sp_tel;
};

// WTA of pixel p from its final sums, W2 u16x2 words in shared memory (16-byte aligned, changed by the
// scan), run by one lane (wta_impl, src/sgm_optimizer.cpp:465-536): the first minimum, the second minimum outside
// |d - best| <= 1, the sub-pixel step.  Every sum carries BIAS; sums >= INF are invalid.  A negative
// winning disparity reads as "none" like the reference's best_d < 0 test (:490-495).
template <int W2, uint32_t INF, uint32_t BIAS>
__device__ __forceinline__ void wta_row(const WtaOut& o, int d0, int D, uint32_t* row, int p) {
    constexpr int NC = W2 / 4;  // chunks of four words
    const auto halves = [](uint32_t v) { return min(v & 0xFFFFu, v >> 16); };
    // the minimum and the first group of GC chunks that holds it, as one key (minimum << 8 | group)
    constexpr int GC = NC <= 16 ? 1 : NC / 16 + (NC % 16 != 0), NGR = NC / GC;
    static_assert(NGR * GC == NC, "groups cover the row");
    uint32_t key = 0xFFFFFFFFu;
#pragma unroll
    for (int g = 0; g < NGR; ++g) {
        uint32_t v = 0xFFFFFFFFu;
#pragma unroll
        for (int c = 0; c < GC; ++c) {
            const uint4 q = *reinterpret_cast<const uint4*>(row + 4 * (g * GC + c));
            v = __vimin3_u16x2(__vimin3_u16x2(v, q.x, q.y), q.z, q.w);
        }
        key = min(key, halves(v) * 256u + g);
    }
    const uint32_t m = key >> 8;
    float dval = -1.f, fb = __int_as_float(0x7f800000), fs = __int_as_float(0x7f800000);
    if (m < INF) {
        // the first halfword of that group equal to m
        const uint32_t* gr = row + 4 * GC * (key & 0xFFu);
        int bdi = 0;
#pragma unroll
        for (int c = GC - 1; c >= 0; --c) {
            const uint4 q = *reinterpret_cast<const uint4*>(gr + 4 * c);
            const uint32_t v[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int i = 3; i >= 0; --i) {
                if ((v[i] >> 16) == m) bdi = 8 * c + 2 * i + 1;
                if ((v[i] & 0xFFFFu) == m) bdi = 8 * c + 2 * i;
            }
        }
        bdi += 8 * GC * (int)(key & 0xFFu);
        if (d0 + bdi >= 0) {
            // the second minimum outside |d - best| <= 1: those three sums are read, taken out of the
            // row, and the row scanned again
            uint16_t* r16 = reinterpret_cast<uint16_t*>(row);
            const uint32_t cm = bdi > 0 ? r16[bdi - 1] : 0xFFFFu, cp = bdi + 1 < 2 * W2 ? r16[bdi + 1] : 0xFFFFu;
            if (bdi > 0) r16[bdi - 1] = 0xFFFFu;
            r16[bdi] = 0xFFFFu;
            if (bdi + 1 < 2 * W2) r16[bdi + 1] = 0xFFFFu;
            uint32_t s0 = 0xFFFFFFFFu, s1 = 0xFFFFFFFFu;
#pragma unroll
            for (int c = 0; c < NC; c += 2) {
                const uint4 q = *reinterpret_cast<const uint4*>(row + 4 * c);
                const uint4 r = *reinterpret_cast<const uint4*>(row + 4 * c + 4);
                s0 = __vimin3_u16x2(__vimin3_u16x2(s0, q.x, q.y), q.z, q.w);
                s1 = __vimin3_u16x2(__vimin3_u16x2(s1, r.x, r.y), r.z, r.w);
            }
            const uint32_t sec = halves(__vminu2(s0, s1));
            const uint32_t bv = m - BIAS;
            dval = (float)(d0 + bdi);
            if (o.subpixel && bdi > 0 && bdi + 1 < D && cm < INF && cp < INF) {
                // WTA uniqueness (src/sgm_optimizer.cpp:520-525): (second - best) / max(best, 1), read by
                // one of the experimental methods only
                float u = 1.0f;
                if (o.sp_method == 2 && sec < INF) u = __fdiv_rn((float)(sec - m), (float)max(bv, 1u));
                const float fm = (float)(cm - BIAS), f0 = (float)bv, fp = (float)(cp - BIAS);
                dval = __fadd_rn(dval, o.sp_tel ? subpixel_delta_tel(fm, f0, fp, o.sp_method, o.sp_param, u, o.sp_tel)
                                                : subpixel_delta(fm, f0, fp, o.sp_method, o.sp_param, u));
            }
            fb = (float)bv;
            fs = sec >= INF ? __int_as_float(0x7f800000) : (float)(sec - BIAS);
        }
    }
    o.disp[p] = dval;
    o.best[p] = fb;
    o.second[p] = fs;
}

}  // namespace apgcu
