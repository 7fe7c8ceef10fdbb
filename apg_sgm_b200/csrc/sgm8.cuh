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

// WTA of pixel p from its final sums, W2 u16x2 words in shared memory (16-byte aligned), run by one
// lane (wta_impl, src/sgm_optimizer.cpp:465-536): the first minimum, the second minimum outside
// |d - best| <= 1, the sub-pixel step.  Every sum carries BIAS; sums >= INF are invalid.  A negative
// winning disparity reads as "none" like the reference's best_d < 0 test (:490-495).
template <int W2, uint32_t INF, uint32_t BIAS>
__device__ __forceinline__ void wta_row(const WtaOut& o, int d0, int D, const uint32_t* row, int p) {
    // one pass over the row keeps the minimum of each chunk of four or eight words in registers; the
    // first index and the second minimum then read the (at most two) chunks they touch again
    constexpr int CS = W2 >= 128 ? 8 : 4;  // words per chunk (W2 is a multiple of 32)
    constexpr int NC = W2 / CS;
    const auto halves = [](uint32_t v) { return min(v & 0xFFFFu, v >> 16); };
    uint32_t cmin[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        uint32_t v = 0xFFFFFFFFu;
#pragma unroll
        for (int i = 0; i < CS; i += 4) {
            const uint4 q = *reinterpret_cast<const uint4*>(row + c * CS + i);
            v = __vminu2(__vimin3_u16x2(v, q.x, q.y), __vminu2(q.z, q.w));
        }
        cmin[c] = v;
    }
    uint32_t all = cmin[0];
#pragma unroll
    for (int c = 1; c < NC; ++c) all = __vminu2(all, cmin[c]);
    const uint32_t m = halves(all);
    float dval = -1.f, fb = __int_as_float(0x7f800000), fs = __int_as_float(0x7f800000);
    if (m < INF) {
        // the first chunk whose minimum is m, then the first halfword equal to m inside it
        int fc = 0;
#pragma unroll
        for (int c = NC - 1; c >= 0; --c)
            if (halves(cmin[c]) == m) fc = c;
        int bdi = 0;
#pragma unroll
        for (int i = CS - 1; i >= 0; --i) {
            const uint32_t v = row[fc * CS + i];
            if ((v >> 16) == m) bdi = 2 * i + 1;
            if ((v & 0xFFFFu) == m) bdi = 2 * i;
        }
        bdi += 2 * fc * CS;
        if (d0 + bdi >= 0) {
            const uint16_t* r16 = reinterpret_cast<const uint16_t*>(row);
            dval = (float)(d0 + bdi);
            // second minimum outside |d - best| <= 1: chunks without an excluded halfword keep
            // their minimum; the (at most two) chunks with one are read again with those masked
            const int klo = bdi > 0 ? (bdi - 1) >> 1 : 0, khi = min((bdi + 1) >> 1, W2 - 1);
            const int clo = klo / CS, chi = khi / CS;
            uint32_t sec2 = 0xFFFFFFFFu;
#pragma unroll
            for (int c = 0; c < NC; ++c)
                if (c != clo && c != chi) sec2 = __vminu2(sec2, cmin[c]);
            for (int c = clo; c <= chi; ++c) {
#pragma unroll
                for (int i = 0; i < CS; ++i) {
                    const int k = c * CS + i;
                    uint32_t v = row[k];
                    if (abs(2 * k - bdi) <= 1) v |= 0x0000FFFFu;
                    if (abs(2 * k + 1 - bdi) <= 1) v |= 0xFFFF0000u;
                    sec2 = __vminu2(sec2, v);
                }
            }
            const uint32_t sec = halves(sec2);
            const uint32_t bv = m - BIAS;
            if (o.subpixel && bdi > 0 && bdi + 1 < D) {
                const uint32_t cm = r16[bdi - 1], cp = r16[bdi + 1];
                if (cm < INF && cp < INF) {
                    // WTA uniqueness (src/sgm_optimizer.cpp:520-525): (second - best) / max(best, 1)
                    const float u = sec >= INF ? 1.0f : __fdiv_rn((float)(sec - m), (float)max(bv, 1u));
                    const float fm = (float)(cm - BIAS), f0 = (float)bv, fp = (float)(cp - BIAS);
                    dval = __fadd_rn(dval, o.sp_tel ? subpixel_delta_tel(fm, f0, fp, o.sp_method, o.sp_param, u, o.sp_tel)
                                                    : subpixel_delta(fm, f0, fp, o.sp_method, o.sp_param, u));
                }
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
