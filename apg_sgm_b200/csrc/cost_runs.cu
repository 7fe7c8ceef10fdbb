// Matching-cost volume by pixel runs, fused with the horizontal Cross-arm pass and the
// right-image argmin: the form used for the 32-bit census (Fast, Balanced, and HighQuality with the
// prior's per-pixel ranges), up to 256 padded disparities.  Results are those of cost.cu's tile
// kernel, which keeps the 64-bit census and wider ranges; only the division of the work differs:
//
//   * One warp covers the whole disparity range of a run of consecutive staged pixels: lane l owns
//     the WPL = Dp/64 words k = WPL*l .. WPL*l + WPL-1 (the P = 2*WPL disparities P*l .. P*l+P-1)
//     and walks the run one pixel per step.  The right pixel of (x+1, di+1) is the right pixel of
//     (x, di), so each step loads one new right descriptor per lane into a P-entry register window;
//     the left descriptor is the same for the whole warp (broadcast loads of four pixels at a time).
//   * Quantised costs follow CostComputer::compute_volume (src/cost_computer.cpp:247-264): the
//     census and AD terms come from one table t2[ad][pop] = lut_census[pop] + lut_ad[ad] (the
//     reference's first float add, done once per entry), then + lut_grad[g], * scale, + 0.5,
//     truncation and clamp, each float op rounded on its own.  Census-only costs use the host's
//     pre-quantised table.
//   * The horizontal prefix over a run (CostAggregator::aggregate_hv's row pass,
//     src/cost_aggregator.cpp:65-105) is a plain 32-bit running sum of packed words: the
//     difference of two such sums is exact in each 16-bit half when each half's window sum is
//     below 2^16, which the host checks for the arm length and cost_max.  Runs are joined at query
//     time from the per-run totals.
//   * Per-pixel ranges: each staged left pixel carries [lo, hi); a lane turns it into a mask of its
//     P disparities per step, and the aggregation keeps a second running prefix of valid counts
//     (two 8-bit counts per word, exact for windows of at most 255 pixels).
//   * The right-image argmin (wta_right_from_left_volume, src/pipeline.cpp:24-85): right pixel
//     r = x - d0 - di receives (x, di) at step x in lane di/P.  Each lane keeps the running minimum
//     keys (cost << 16 | di: lowest cost first, then lowest d) of its P right pixels; every step
//     the oldest moves one lane up (a shuffle), and the one leaving lane 31 -- complete over this
//     run -- goes to a per-warp buffer; at the end of the run these and the partial minima still
//     held are merged into the tile's keys in shared memory, and those into rkey with one coalesced
//     atomicMin per right pixel of the tile.  min is idempotent, so a halo pixel seen by two tiles
//     changes nothing.
//
// Bound: issue slots and the shared-memory gathers (two table entries per voxel, 3.5 and 2.4 bank passes a
// warp on textured frames), then the population count (eight cycles a warp instruction).  Merging the keys in
// shared memory, testing validity by two packed compares per word and walking the tiles by columns took the
// kernel from 439 to 239 us (Fast 1920x1080 D256), 267 to 250 (Balanced 1280x720 D128), 264 to 235 (997x611).
// Table addresses by dot products, with the table's base as the addend: 250 to 243, 235 to 224.
// Where the ranges are narrow (the coarse pass leaves about 10 of 128 disparities a pixel), 64 disparities a run
// and quads by range: hierarchical 1280x720 D128 362 -> 268 us, HighQuality 1920x1080 D256 1466 -> 1437.
//
// Blocks are persistent: each builds its tables once and then walks (row, column tile) items.
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "kernels.h"

namespace apgcu {

namespace {

// t2[pop][|dgray|]: one row of 256 per popcount 0..32 of a 32-bit census, so a voxel's index is
// one byte permute of the popcount and the absolute differences
constexpr int kT2Rows = 33;

struct RunGeom {
    int txc, ha, nx, nr, roff, rl, nrun, ntx, ntiles;
    size_t t2, lgt, q, magic, arm, lc, lg, rc, rg, rng, pre, cnt, tot, totc, emit, key, total;
};

inline size_t a16(size_t v) { return (v + 15) & ~size_t(15); }

inline int run_warps(bool cross) { return cross ? 16 : 8; }

// Staging and table layout of one block for a tile of txc columns with halo ha.  nx (staged left
// pixels) and rl (run length) are multiples of 4 (16-byte loads of four left descriptors); roff
// shifts the staged right row so that each step group's right descriptors start at a multiple of four
// (16-byte loads) or, with 64 or 192 padded disparities, an even index (8-byte loads) and every lane with a disparity inside the range finds its whole window staged.
// One run per warp.
RunGeom run_geom(const CostCtx& c, int txc, int ha, bool cross, bool full, bool prior) {
    RunGeom g{};
    const int W2 = c.Dp / 2;
    g.txc = txc;
    g.ha = ha;
    g.nrun = run_warps(cross);
    g.nx = round_up(txc + 2 * ha, 4);
    g.rl = round_up((g.nx + g.nrun - 1) / g.nrun, 4);
    // aligned start for every step group (of four entries where P is a multiple of four, else of two),
    // plus P entries so that a lane holding any disparity of the range loads its own window without
    // clamping
    const int P = c.Dp / 32;
    g.roff = (P % 4 == 0 ? (4 - (c.D - 1) % 4) % 4 : ((c.D - 1) % 2 == 0 ? 2 : 1)) + P;
    g.nr = round_up(g.nx + c.D - 1 + g.roff, 4);
    g.ntx = (c.w + txc - 1) / txc;
    g.ntiles = g.ntx * c.h;
    const bool stage_g = full || cross;
    size_t o = 0;
    g.t2 = o; o = a16(o + (full ? 256 * kT2Rows * 4 : 0));
    g.lgt = o; o = a16(o + (full ? 511 * 4 : 0));
    g.q = o; o = a16(o + (full ? 0 : 65 * 4));
    g.magic = o; o = a16(o + (cross ? (2 * ha + 2) * 4 : 0));
    g.arm = o; o = a16(o + (cross ? txc * 4 : 0));
    g.lc = o; o = a16(o + g.nx * 4);
    g.lg = o; o = a16(o + (stage_g ? g.nx * 4 : 0));
    g.rc = o; o = a16(o + g.nr * 4);
    g.rg = o; o = a16(o + (full ? g.nr * 4 : 0));
    g.rng = o; o = a16(o + (prior ? g.nx * 4 : 0));                                // lo | hi << 16
    g.pre = o; o = a16(o + (cross ? (size_t)g.nx * W2 * 4 : 0));
    g.cnt = o; o = a16(o + (cross && prior ? (size_t)g.nx * W2 * 2 : 0));        // valid counts
    g.tot = o; o = a16(o + (cross ? (size_t)g.nrun * W2 * 4 : 0));
    g.totc = o; o = a16(o + (cross && prior ? (size_t)g.nrun * W2 * 2 : 0));
    g.emit = o; o = a16(o + (size_t)g.nrun * g.rl * 4);
    g.key = o; o = a16(o + (size_t)(g.nx + c.Dp) * 4);  // argmin keys of the tile's right pixels
    g.total = o;
    return g;
}

__device__ __forceinline__ uint32_t pack_g(const uint8_t* gray, const uint8_t* gx, const uint8_t* gy, int i) {
    return (uint32_t)gray[i] | ((uint32_t)gx[i] << 8) | ((uint32_t)gy[i] << 16);
}

// Quantised costs of two (left, right) descriptor pairs (disparities 2w and 2w + 1 of one lane),
// packed low / high: the reference's float steps (src/cost_computer.cpp:247-264), each rounded on
// its own, two lanes per packed f32x2 instruction.  (int)(v * scale + 0.5f) truncates a value in
// [0.5, 2^23): adding 2^23 rounded toward zero leaves exactly 2^23 + trunc(v), so the integer is
// the low mantissa bits; truncation saturates below zero in the reference, and here v >= 0.5.
__device__ __forceinline__ unsigned long long f2add_rn(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long f2add_rz(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("add.rz.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long f2mul_rn(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long f2pack(float lo, float hi) {
    return (unsigned long long)__float_as_uint(lo) | ((unsigned long long)__float_as_uint(hi) << 32);
}

// 0xFFFF in each half whose top bit is set (the permute's sign mode: bytes 1 and 3), else 0
__device__ __forceinline__ uint32_t spread_top_bits(uint32_t v) {
    uint32_t r;
    asm("prmt.b32 %0, %1, 0, 0xBB99;" : "=r"(r) : "r"(v));
    return r;
}

__device__ __forceinline__ float lds_f32(uint32_t a) {
    float v;
    asm("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
}

template <bool FULL>
__device__ __forceinline__ uint32_t run_cost2(uint32_t lc, uint32_t lg, uint32_t rc0, uint32_t rg0, uint32_t rc1,
                                              uint32_t rg1, const float* s_t2, const float* s_lgt,
                                              const uint32_t* s_q, unsigned long long scale2, uint32_t cmax2) {
    const uint32_t pop0 = __popc(lc ^ rc0), pop1 = __popc(lc ^ rc1);
    if constexpr (!FULL) {
        return __byte_perm(s_q[pop0], s_q[pop1], 0x5410);
    } else {
        const uint32_t ad0 = __vabsdiffu4(lg, rg0), ad1 = __vabsdiffu4(lg, rg1);  // |dgray|, |dgx|, |dgy|
        // byte addresses by dot products: t2[pop][|dgray|] at pop * 1024 + 4 |dgray|, lut_grad at 4 (|dgx| + |dgy|)
        const uint32_t bt = (uint32_t)__cvta_generic_to_shared(s_t2), bg = (uint32_t)__cvta_generic_to_shared(s_lgt);
        const float t0 = lds_f32(__dp4a(ad0, 0x00000004u, bt) + (pop0 << 10));
        const float t1 = lds_f32(__dp4a(ad1, 0x00000004u, bt) + (pop1 << 10));
        const float g0 = lds_f32(__dp4a(ad0, 0x00040400u, bg));
        const float g1 = lds_f32(__dp4a(ad1, 0x00040400u, bg));
        const unsigned long long v = f2add_rn(f2pack(t0, t1), f2pack(g0, g1));
        const unsigned long long u = f2add_rn(f2mul_rn(v, scale2), 0x3F0000003F000000ull);  // + 0.5f
        const unsigned long long q = f2add_rz(u, 0x4B0000004B000000ull);                    // + 2^23, toward 0
        // the low 16 bits of each lane's mantissa are its integer (< 2^16 by the host's cost_max check)
        return __vminu2(__byte_perm((uint32_t)q, (uint32_t)(q >> 32), 0x5410), cmax2);
    }
}

template <int N>
__device__ __forceinline__ void store_words(uint32_t* p, const uint32_t (&w)[N]) {
    if constexpr (N == 4) {
        *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
    } else if constexpr (N == 2) {
        *reinterpret_cast<uint2*>(p) = make_uint2(w[0], w[1]);
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) p[i] = w[i];
    }
}

// WPL 16-bit count words (two 8-bit valid counts each) at p, which is 4-byte aligned for even WPL.
template <int N>
__device__ __forceinline__ void store_counts(uint16_t* p, const uint32_t (&c)[N]) {
    if constexpr (N % 2 == 0) {
#pragma unroll
        for (int i = 0; i < N; i += 2)
            *reinterpret_cast<uint32_t*>(p + i) = (c[i] & 0xFFFFu) | (c[i + 1] << 16);
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) p[i] = (uint16_t)c[i];
    }
}

// One run of steps of this lane's P disparities.  V: every (x, d) of the run is a valid voxel for
// every lane of the warp (no per-voxel tests).
// PRIOR: every left pixel has its own range [lo, hi) (staged in s_rng); a voxel outside it is
// invalid, and the aggregation also keeps a prefix of valid counts (s_cnt, s_totc).
// W2: words per pixel of the volume.  The lanes' words start at kb (0 where the warp covers them all).
template <bool V, bool CROSS, bool STORE, bool FULL, int WPL, int W2, bool PRIOR, bool U8>
__device__ __forceinline__ void run_steps(const CostCtx& c, const RunGeom& g, int row, int xbase, int xs, int xe,
                                          const uint32_t* s_lc, const uint32_t* s_lg, const uint32_t* s_rc,
                                          const uint32_t* s_rg, const float* s_t2, const float* s_lgt,
                                          const uint32_t* s_q, const uint32_t* s_rng, uint32_t* s_pre,
                                          uint16_t* s_cnt, uint32_t* s_tot, uint16_t* s_totc, uint32_t* s_em,
                                          uint32_t* s_key, int run, int kb, uint32_t* __restrict__ out_vol) {
    constexpr int P = 2 * WPL;
    const int lane = threadIdx.x & 31;
    const int dbase = P * lane + 2 * kb;  // first disparity index of this lane
    const unsigned long long scale2 = f2pack(c.scale, c.scale);
    const uint32_t cmax2 = (uint32_t)c.cost_max * 0x00010001u;
    // a step group's four right descriptors in one load where the lanes' windows allow it: at a stride of
    // P words, two 8-byte loads would hit every bank twice as often
    constexpr bool kWide = P % 4 == 0;
    // lanes wholly past the range load at the last in-bounds aligned base (dl + P <= D + roff keeps
    // every window entry inside the staged row) and are masked; a lane with any disparity below D has
    // dbase <= D - 1 < D + roff - P (rounded down to the alignment too), so keeps its own
    const int dl = V ? dbase : min(dbase, (c.D + g.roff - P) & (kWide ? ~3 : ~1));
    int ri = xs - dl + c.D - 1 + g.roff;  // staged right descriptor of (xs, dl); aligned
    uint32_t wc[P], wg[P], acc[P], pre[WPL], cnt[WPL];
#pragma unroll
    for (int j = 0; j < P; ++j) {
        // before the first step's shift: wc[j] holds the descriptor of (xs - 1, dl + j)
        wc[j] = j < P - 1 ? s_rc[ri - 1 - j] : 0u;
        wg[j] = (FULL && j < P - 1) ? s_rg[ri - 1 - j] : 0u;
        acc[j] = kInvalidWord;
    }
#pragma unroll
    for (int w = 0; w < WPL; ++w) pre[w] = cnt[w] = 0;
    uint32_t* pp = s_pre + xs * W2 + kb + WPL * lane;                             // prefix words of (xs)
    uint16_t* cp = s_cnt + xs * W2 + kb + WPL * lane;                             // count words of (xs)
    uint32_t* vp = out_vol + ((size_t)row + (xbase + xs)) * W2 + WPL * lane;  // volume words of (xs)
    // byte volume: the lane's P disparities of (xs)
    uint8_t* vp8 = reinterpret_cast<uint8_t*>(out_vol) + ((size_t)row + (xbase + xs)) * (2 * W2) + P * lane;
    for (int xi = xs; xi < xe; xi += 4) {
        const uint4 lc4 = *reinterpret_cast<const uint4*>(s_lc + xi);
        uint4 lg4 = make_uint4(0, 0, 0, 0);
        if (FULL) lg4 = *reinterpret_cast<const uint4*>(s_lg + xi);
        uint2 na, nb, ga = make_uint2(0, 0), gb = make_uint2(0, 0);
        if constexpr (kWide) {
            const uint4 nc = *reinterpret_cast<const uint4*>(s_rc + ri);
            na = make_uint2(nc.x, nc.y);
            nb = make_uint2(nc.z, nc.w);
            if (FULL) {
                const uint4 ng = *reinterpret_cast<const uint4*>(s_rg + ri);
                ga = make_uint2(ng.x, ng.y);
                gb = make_uint2(ng.z, ng.w);
            }
        } else {
            na = *reinterpret_cast<const uint2*>(s_rc + ri);
            nb = *reinterpret_cast<const uint2*>(s_rc + ri + 2);
            if (FULL) {
                ga = *reinterpret_cast<const uint2*>(s_rg + ri);
                gb = *reinterpret_cast<const uint2*>(s_rg + ri + 2);
            }
        }
        uint32_t em[4];
        const uint32_t L[4] = {lc4.x, lc4.y, lc4.z, lc4.w};
        const uint32_t LG[4] = {lg4.x, lg4.y, lg4.z, lg4.w};
        const uint32_t NC[4] = {na.x, na.y, nb.x, nb.y};
        const uint32_t NG[4] = {ga.x, ga.y, gb.x, gb.y};
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const int x = xbase + xi + s;
#pragma unroll
            for (int j = P - 1; j > 0; --j) {
                wc[j] = wc[j - 1];
                wg[j] = wg[j - 1];
            }
            wc[0] = NC[s];
            wg[0] = NG[s];
            uint32_t qp[WPL];  // quantised costs of disparities 2w | 2w + 1 << 16
            uint32_t vm[WPL];  // their validity: 0xFFFF per valid half
            // this lane's valid disparities [lo, hi) of the pixel: inside its own range (PRIOR), inside
            // the image and the range (!V).  Both bounds in both halves, biased so that a difference's
            // top bit is the comparison's outcome
            uint32_t lo2 = 0, hi2 = 0;
            if (!V || PRIOR) {
                int lo = 0, hi = P;
                if (PRIOR) {
                    const uint32_t rg = s_rng[xi + s];
                    const int base = c.d0 + dbase;
                    lo = (int)(int16_t)(rg & 0xFFFFu) - base;
                    hi = (int)(int16_t)(rg >> 16) - base;
                }
                if (!V) {
                    const int xd = x - c.d0 - dbase;  // right column of the lane's first disparity
                    lo = max(lo, xd - (c.w - 1));
                    hi = min(min(hi, xd + 1), c.D - dbase);
                    if (x < 0 || x >= c.w) hi = 0;
                }
                lo2 = (uint32_t)min(max(lo, 0), P) * 0x00010001u;
                hi2 = (uint32_t)min(max(hi, 0), P) * 0x00010001u + 0x7FFF7FFFu;
            }
#pragma unroll
            for (int w = 0; w < WPL; ++w) {
                qp[w] = run_cost2<FULL>(L[s], LG[s], wc[2 * w], wg[2 * w], wc[2 * w + 1], wg[2 * w + 1], s_t2, s_lgt,
                                        s_q, scale2, cmax2);
                vm[w] = 0xFFFFFFFFu;
                uint32_t qk = qp[w];
                if (!V || PRIOR) {
                    const uint32_t jp = (uint32_t)(2 * w) | ((uint32_t)(2 * w + 1) << 16);
                    // top bit of each half: j >= lo and j < hi, spread over the half
                    vm[w] = spread_top_bits(((jp | 0x80008000u) - lo2) & (hi2 - jp));
                    qk |= ~vm[w];
                }
                // keys (cost << 16 | disparity index); an invalid voxel's is 0xFFFF0000 or more, above any cost
                acc[2 * w] = min(acc[2 * w], (qk << 16) | (uint32_t)(dbase + 2 * w));
                acc[2 * w + 1] = min(acc[2 * w + 1], (qk & 0xFFFF0000u) | (uint32_t)(dbase + 2 * w + 1));
            }
            // the oldest minimum moves one lane up; lane 31's is complete for this run
            const uint32_t out = acc[P - 1];
            em[s] = out;
            const uint32_t in = __shfl_up_sync(0xFFFFFFFFu, out, 1);
#pragma unroll
            for (int j = P - 1; j > 0; --j) acc[j] = acc[j - 1];
            acc[0] = lane ? in : kInvalidWord;
            if (CROSS) {
#pragma unroll
                for (int w = 0; w < WPL; ++w) pre[w] += qp[w] & vm[w];
                store_words<WPL>(pp + s * W2, pre);
                if (PRIOR) {
#pragma unroll
                    for (int w = 0; w < WPL; ++w) cnt[w] += __byte_perm(vm[w], 0u, 0x4420) & 0x0101u;  // (valid low) | (valid high) << 8
                    store_counts<WPL>(cp + s * W2, cnt);
                }
            } else if (STORE) {
                // without a halo the staged pixels are the tile's; V runs lie inside the image
                if (V || (xi + s < g.txc && x < c.w)) {
                    uint32_t wd[WPL];
#pragma unroll
                    for (int w = 0; w < WPL; ++w) wd[w] = qp[w] | ~vm[w];  // invalid halves: 0xFFFF
                    if constexpr (U8) {
                        // the low byte of each half: costs are below 255, the invalid 0xFFFF becomes 0xFF
                        if constexpr (WPL % 2 == 0) {
                            uint32_t wb[WPL / 2];
#pragma unroll
                            for (int w = 0; w < WPL / 2; ++w) wb[w] = __byte_perm(wd[2 * w], wd[2 * w + 1], 0x6420);
                            store_words<WPL / 2>(reinterpret_cast<uint32_t*>(vp8 + (size_t)s * (2 * W2)), wb);
                        } else {
#pragma unroll
                            for (int w = 0; w < WPL; ++w)
                                *reinterpret_cast<uint16_t*>(vp8 + (size_t)s * (2 * W2) + 2 * w) =
                                    (uint16_t)__byte_perm(wd[w], 0u, 0x4420);
                        }
                    } else {
                        store_words<WPL>(vp + (size_t)s * W2, wd);
                    }
                }
            }
        }
        if (lane == 31) *reinterpret_cast<uint4*>(s_em + (xi - xs)) = make_uint4(em[0], em[1], em[2], em[3]);
        ri += 4;
        pp += 4 * W2;
        cp += 4 * W2;
        vp += 4 * (size_t)W2;
        vp8 += 8 * (size_t)W2;
    }
    __syncwarp();
    if (xe > xs) {
        // into the tile's keys (index 0: right pixel xbase - d0 - (Dp - 1)): the minima that left lane 31 at
        // step xs + e, and the partial ones still held (acc[j] is of right pixel xbase + xe - d0 - dbase - j)
        const int n = xe - xs;
        uint32_t* ke = s_key + xs + 2 * (W2 - 32 * WPL - kb);
        for (int e = lane; e < n; e += 32)
            if (s_em[e] < 0xFFFF0000u) atomicMin(ke + e, s_em[e]);
        uint32_t* kp = s_key + xe - dbase + 2 * W2 - 1;
#pragma unroll
        for (int j = 0; j < P; ++j)
            if (acc[j] < 0xFFFF0000u) atomicMin(kp - j, acc[j]);
    }
    __syncwarp();
    if (CROSS) store_words<WPL>(s_tot + run * W2 + kb + WPL * lane, pre);
    if (CROSS && PRIOR) store_counts<WPL>(s_totc + run * W2 + kb + WPL * lane, cnt);
}

// floor(s / n) of a window sum and its count, by the table's reciprocal m of n: 2^32 / n (div_by_magic),
// or, for the byte output (costs of at most 254), 2^24 / n, the quotient in the product's top byte (the
// bound is derived in cross8.cu).
template <bool U8>
__device__ __forceinline__ uint32_t window_div(uint32_t s, uint32_t n, uint32_t m) {
    if constexpr (U8) return (s * m) >> 24;
    else return div_by_magic(s, n, m);
}

// Aggregated word kk at pixel x from its packed window sum s (cost.cu's tile kernel, same rules).
template <bool U8>
__device__ __forceinline__ uint32_t agg_word(const CostCtx& c, uint32_t s, int kk, int x, int l, int r,
                                             const uint32_t* s_magic) {
    const int dw = c.d0 + 2 * kk;
    if (2 * kk + 1 < c.D && x - l >= dw + 1 && x + r <= c.w - 1 + dw) {
        const uint32_t len = (uint32_t)(l + r + 1), mg = s_magic[len];
        return window_div<U8>(s & 0xFFFFu, len, mg) | (window_div<U8>(s >> 16, len, mg) << 16);
    }
    uint32_t word = 0;
#pragma unroll
    for (int hs = 0; hs < 2; ++hs) {
        const int di = 2 * kk + hs;
        const int d = c.d0 + di;
        const uint32_t sh = (s >> (16 * hs)) & 0xFFFFu;
        const int nh = min(x + r, c.w - 1 + d) - max(x - l, d) + 1;  // valid x' in the window
        const bool ok = di < c.D && d <= x && nh > 0;
        const uint32_t q = ok ? window_div<U8>(sh, (uint32_t)nh, s_magic[nh]) : kInvalidCost;
        word |= q << (16 * hs);
    }
    return word;
}

// Aggregated word kk from its window sum s and its two 8-bit valid counts n, with per-pixel ranges
// (cost.cu's tile kernel, same rule): a half is valid when its disparity is inside the centre
// pixel's range and its window holds a valid voxel.
template <bool U8>
__device__ __forceinline__ uint32_t prior_word(const CostCtx& c, uint32_t s, uint32_t n, int kk, int lo, int hi,
                                               const uint32_t* s_magic) {
    uint32_t word = 0;
#pragma unroll
    for (int hs = 0; hs < 2; ++hs) {
        const int di = 2 * kk + hs;
        const int d = c.d0 + di;
        const uint32_t sh = (s >> (16 * hs)) & 0xFFFFu, nh = (n >> (8 * hs)) & 0xFFu;
        const bool ok = di < c.D && d >= lo && d < hi && nh > 0;
        const uint32_t q = ok ? window_div<U8>(sh, nh, s_magic[nh]) : kInvalidCost;
        word |= q << (16 * hs);
    }
    return word;
}

// With 192 or 256 padded disparities the aggregating kernel keeps one block per SM (registers for
// the wider lane state, wider tiles: less halo); otherwise two.
template <bool CROSS, bool STORE, bool FULL, int WPL, bool PRIOR, bool U8>
__global__ void __launch_bounds__(CROSS ? 512 : 256, CROSS ? (WPL > 2 ? 1 : 2) : 1)
    cost_run_kernel(CostCtx c, RunGeom g, int lmax, int tau, uint32_t* __restrict__ out_vol,
                    uint32_t* __restrict__ rkey, const uint32_t* __restrict__ magic) {
    constexpr int W2 = 32 * WPL;
    constexpr int P = 2 * WPL;
    extern __shared__ __align__(16) unsigned char smem[];
    float* s_t2 = reinterpret_cast<float*>(smem + g.t2);
    float* s_lgt = reinterpret_cast<float*>(smem + g.lgt);
    uint32_t* s_q = reinterpret_cast<uint32_t*>(smem + g.q);
    uint32_t* s_magic = reinterpret_cast<uint32_t*>(smem + g.magic);
    uint32_t* s_arm = reinterpret_cast<uint32_t*>(smem + g.arm);
    uint32_t* s_lc = reinterpret_cast<uint32_t*>(smem + g.lc);
    uint32_t* s_lg = reinterpret_cast<uint32_t*>(smem + g.lg);
    uint32_t* s_rc = reinterpret_cast<uint32_t*>(smem + g.rc);
    uint32_t* s_rg = reinterpret_cast<uint32_t*>(smem + g.rg);
    uint32_t* s_pre = reinterpret_cast<uint32_t*>(smem + g.pre);
    uint32_t* s_tot = reinterpret_cast<uint32_t*>(smem + g.tot);
    uint32_t* s_rng = reinterpret_cast<uint32_t*>(smem + g.rng);
    uint16_t* s_cnt = reinterpret_cast<uint16_t*>(smem + g.cnt);
    uint16_t* s_totc = reinterpret_cast<uint16_t*>(smem + g.totc);
    const int tid = threadIdx.x, nt = blockDim.x, run = tid >> 5, lane = tid & 31;
    uint32_t* s_em = reinterpret_cast<uint32_t*>(smem + g.emit) + run * g.rl;
    uint32_t* s_key = reinterpret_cast<uint32_t*>(smem + g.key);

    if (FULL) {
        for (int i = tid; i < 256 * kT2Rows; i += nt) {
            const int pop = i >> 8, ad = i & 255;
            const float lc = c.lut[kLutCensus + pop];
            s_t2[i] = c.use_ad ? __fadd_rn(lc, c.lut[kLutAd + ad]) : lc;
        }
        // without the gradient term, + 0.0f leaves every sum as it is
        for (int i = tid; i < 511; i += nt) s_lgt[i] = c.use_grad ? c.lut[kLutGrad + i] : 0.0f;
    } else {
        for (int i = tid; i < 65; i += nt) s_q[i] = c.qlut[i];
    }
    if (CROSS)
        for (int i = tid; i < 2 * g.ha + 2; i += nt) s_magic[i] = U8 ? (i ? (1u << 24) / (uint32_t)i + 1u : 0u) : magic[i];

    const int xs = min(run * g.rl, g.nx), xe = min(xs + g.rl, g.nx);

    for (int tile = blockIdx.x; tile < g.ntiles; tile += gridDim.x) {
        // column by column: the left ones, whose voxels reach out of the image and are tested one by one,
        // then fall on every block alike (row by row, a number of blocks divisible by the tiles of a row
        // gave them all to the same blocks: Fast 1920x1080 D256 in four tiles, 287 us)
        const int col = tile / c.h;
        const int y = tile - col * c.h;
        const int x0 = col * g.txc;
        const int xbase = x0 - g.ha;
        const int rbase = xbase - (c.d0 + c.D - 1) - g.roff;  // image column of staged right 0
        const int row = y * c.w;
        __syncthreads();  // the previous item's readers are done with the staging
        for (int i = tid; i < g.nx + c.Dp; i += nt) s_key[i] = kInvalidWord;
        for (int i = tid; i < g.nx; i += nt) {
            const int x = xbase + i;
            const bool in = x >= 0 && x < c.w;
            s_lc[i] = in ? c.cl[row + x] : 0u;
            if (FULL || CROSS) s_lg[i] = in ? pack_g(c.lgray, c.lgx, c.lgy, row + x) : 0u;
            // outside the image: an empty range
            if (PRIOR) s_rng[i] = in ? ((uint32_t)(uint16_t)c.rmin[row + x] | ((uint32_t)(uint16_t)c.rmax[row + x] << 16)) : 0u;
        }
        for (int i = tid; i < g.nr; i += nt) {
            const int xr = rbase + i;
            const bool in = xr >= 0 && xr < c.w;
            s_rc[i] = in ? c.cr[row + xr] : 0u;
            if (FULL) s_rg[i] = in ? pack_g(c.rgray, c.rgx, c.rgy, row + xr) : 0u;
        }
        __syncthreads();
        if (CROSS) {
            // arms (build_cross_arms, src/cost_aggregator.cpp:17-63) and the runs each window
            // spans: l | r << 8 | run(a - 1) << 16 | run(b) << 24 over staged [a, b]
            for (int i = tid; i < g.txc; i += nt) {
                const int x = x0 + i;
                if (x >= c.w) break;
                const int sxi = i + g.ha;
                const int c0 = (int)(s_lg[sxi] & 0xFFu);
                int l = 0, r = 0;
                while (l < lmax && x - l - 1 >= 0 && abs((int)(s_lg[sxi - l - 1] & 0xFFu) - c0) <= tau) ++l;
                while (r < lmax && x + r + 1 < c.w && abs((int)(s_lg[sxi + r + 1] & 0xFFu) - c0) <= tau) ++r;
                const int a = sxi - l, b = sxi + r;
                const int rlo = a > 0 ? (a - 1) / g.rl : 0, rhi = b / g.rl;
                s_arm[i] = (uint32_t)l | ((uint32_t)r << 8) | ((uint32_t)rlo << 16) | ((uint32_t)rhi << 24);
            }
        }
        // Per-pixel ranges: a run whose pixels' ranges lie in 64 disparities (32 words from kb) is walked with
        // two disparities a lane; its other words' prefixes, counts and totals are zero.
        bool narrow = false;
        if constexpr (CROSS && PRIOR && WPL > 1) {
            unsigned ul = 0xFFFFu, uh = 0;
            for (int i = xs + lane; i < xe; i += 32) {
                const uint32_t rg = s_rng[i];
                const int lo = max((int)(int16_t)(rg & 0xFFFFu) - c.d0, 0), hi = min((int)(int16_t)(rg >> 16) - c.d0, c.D);
                if (lo < hi) {
                    ul = min(ul, (unsigned)lo);
                    uh = max(uh, (unsigned)hi);
                }
            }
            ul = __reduce_min_sync(0xFFFFFFFFu, ul);
            uh = __reduce_max_sync(0xFFFFFFFFu, uh);
            const int kb = min((int)(ul >> 1) & ~3, W2 - 32);  // no valid voxel: uh = 0
            narrow = (int)uh <= 2 * kb + 64;
            if (narrow) {
                run_steps<false, CROSS, STORE, FULL, 1, W2, PRIOR, U8>(c, g, row, xbase, xs, xe, s_lc, s_lg, s_rc, s_rg,
                                                                   s_t2, s_lgt, s_q, s_rng, s_pre, s_cnt, s_tot,
                                                                   s_totc, s_em, s_key, run, kb, out_vol);
                constexpr int zq = (W2 - 32) / 4;
                for (int i = lane; i < (xe - xs + 1) * zq; i += 32) {
                    const int px = i / zq, q4 = 4 * (i - px * zq);
                    const int k4 = q4 < kb ? q4 : q4 + 32;
                    // the row past the last pixel: the run's totals
                    uint32_t* zp = px < xe - xs ? s_pre + (xs + px) * W2 : s_tot + run * W2;
                    uint16_t* zc = px < xe - xs ? s_cnt + (xs + px) * W2 : s_totc + run * W2;
                    *reinterpret_cast<uint4*>(zp + k4) = make_uint4(0, 0, 0, 0);
                    *reinterpret_cast<uint2*>(zc + k4) = make_uint2(0, 0);
                }
            }
        }
        if (!narrow) {
            const int xa = xbase + xs, xb = xbase + xe - 1;
            const int dlo = c.d0 + P * lane;
            const bool ok = xa >= 0 && xb < c.w && P * lane + P - 1 < c.D && xa - (dlo + P - 1) >= 0 &&
                            xb - dlo <= c.w - 1;
            if (__all_sync(0xFFFFFFFFu, ok))
                run_steps<true, CROSS, STORE, FULL, WPL, W2, PRIOR, U8>(c, g, row, xbase, xs, xe, s_lc, s_lg, s_rc, s_rg,
                                                                    s_t2, s_lgt, s_q, s_rng, s_pre, s_cnt, s_tot,
                                                                    s_totc, s_em, s_key, run, 0, out_vol);
            else
                run_steps<false, CROSS, STORE, FULL, WPL, W2, PRIOR, U8>(c, g, row, xbase, xs, xe, s_lc, s_lg, s_rc, s_rg,
                                                                     s_t2, s_lgt, s_q, s_rng, s_pre, s_cnt, s_tot,
                                                                     s_totc, s_em, s_key, run, 0, out_vol);
        }
        // most runs of the tile narrow: the output pass goes by the pixels' ranges too
        bool sparse = false;
        if constexpr (CROSS && PRIOR && WPL > 1) sparse = 4 * __syncthreads_count(narrow) >= 3 * nt;
        else __syncthreads();
        {
            // the tile's keys (from the last thread down: the first ones scan the run offsets)
            const int r0 = xbase - c.d0 - (c.Dp - 1);
            for (int i = nt - 1 - tid; i < g.nx + c.Dp; i += nt) {
                const uint32_t m = s_key[i];
                const int r = r0 + i;
                if (m != kInvalidWord && r >= 0 && r < c.w) atomicMin(rkey + row + r, m);
            }
        }
        if (CROSS) {
            // run offsets: the run totals become an exclusive prefix over the runs, per word, so a
            // window's sum is two lookups whatever number of runs it spans (sums wrap modulo 2^32
            // and counts modulo 2^16; the window differences are exact, as for the prefixes)
            for (int k = tid; k < W2; k += nt) {
                uint32_t acc = 0;
                for (int j = 0; j < g.nrun; ++j) {
                    const uint32_t v = s_tot[j * W2 + k];
                    s_tot[j * W2 + k] = acc;
                    acc += v;
                }
                if (PRIOR) {
                    uint16_t accc = 0;
                    for (int j = 0; j < g.nrun; ++j) {
                        const uint16_t v = s_totc[j * W2 + k];
                        s_totc[j * W2 + k] = accc;
                        accc = (uint16_t)(accc + v);
                    }
                }
            }
            __syncthreads();
            // T(x, d) = floor(window sum / valid count) over [x - L(x), x + R(x)]; a thread takes
            // four words of one pixel, so the pixel's arms, divisor and border tests serve eight
            // disparities and its loads are independent
            constexpr int quads = W2 / 4;
            // In a tile of narrow ranges only a pixel's quads that meet its range are worked out; the others are
            // filled.  Each warp takes a share of the pixels and deals their quads to its lanes.
            const int share = (g.txc + g.nrun - 1) / g.nrun;  // at most 32 (cross_tile)
            int items = g.txc * quads, step = nt, first = tid, px = 0, q0 = 0, upto = 0;
            if (sparse) {
                for (int i = tid; i < g.txc * quads; i += nt) {
                    const int xi = i / quads, k4 = 4 * (i - xi * quads);
                    if (x0 + xi >= c.w) break;
                    const uint32_t rg = s_rng[xi + g.ha];
                    const int lo = (int)(int16_t)(rg & 0xFFFFu) - c.d0, hi = (int)(int16_t)(rg >> 16) - c.d0;
                    if (lo < hi && 2 * k4 + 8 > lo && 2 * k4 < hi) continue;
                    if constexpr (U8)
                        *reinterpret_cast<uint2*>(reinterpret_cast<uint8_t*>(out_vol) + ((size_t)row + x0 + xi) * (2 * W2) + 2 * k4) =
                            make_uint2(0xFFFFFFFFu, 0xFFFFFFFFu);
                    else
                        *reinterpret_cast<uint4*>(out_vol + ((size_t)row + x0 + xi) * W2 + k4) =
                            make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu);
                }
                // this lane's pixel of the share: its first quad, and the running total of quads
                px = run * share + lane;
                int nq = 0;
                if (lane < share && px < g.txc && x0 + px < c.w) {
                    const uint32_t rg = s_rng[px + g.ha];
                    const int lo = max((int)(int16_t)(rg & 0xFFFFu) - c.d0, 0);
                    const int hi = min((int)(int16_t)(rg >> 16) - c.d0, 8 * quads);
                    if (lo < hi) {
                        q0 = lo >> 3;
                        nq = ((hi - 1) >> 3) - q0 + 1;
                    }
                }
                upto = nq;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xFFFFFFFFu, upto, o);
                    if (lane >= o) upto += v;
                }
                q0 -= upto - nq;  // so that item i of the pixel is quad q0 + i
                items = __shfl_sync(0xFFFFFFFFu, upto, 31);
                items = (items + 31) & ~31;  // whole warps: the owners' search shuffles
                step = 32;
                first = lane;
            }
            for (int item = first; item < items; item += step) {
                int xi, k4;
                if (sparse) {
                    // the owner: the first lane whose running total exceeds the item
                    int o = 0;
#pragma unroll
                    for (int b = 16; b; b >>= 1)
                        if (__shfl_sync(0xFFFFFFFFu, upto, o + b - 1) <= item) o += b;
                    const int oq = __shfl_sync(0xFFFFFFFFu, q0, o);
                    if (item >= __shfl_sync(0xFFFFFFFFu, upto, 31)) continue;
                    xi = run * share + o;
                    k4 = 4 * (oq + item);
                } else {
                    xi = item / quads;
                    k4 = 4 * (item - xi * quads);
                }
                const int x = x0 + xi;
                if (x >= c.w) break;
                const uint32_t arm = s_arm[xi];
                const int l = (int)(arm & 0xFFu), r = (int)((arm >> 8) & 0xFFu);
                const int rlo = (int)((arm >> 16) & 0xFFu), rhi = (int)(arm >> 24);
                const int sxi = xi + g.ha, a = sxi - l, b = sxi + r;
                const uint4 pb = *reinterpret_cast<const uint4*>(s_pre + b * W2 + k4);
                // the offsets of the runs at the window's ends cancel where it lies in one run
                uint4 ob = make_uint4(0, 0, 0, 0), oa = ob;
                if (rhi != rlo) {
                    ob = *reinterpret_cast<const uint4*>(s_tot + rhi * W2 + k4);
                    oa = *reinterpret_cast<const uint4*>(s_tot + rlo * W2 + k4);
                }
                const uint4 pa = a > 0 ? *reinterpret_cast<const uint4*>(s_pre + (a - 1) * W2 + k4) : make_uint4(0, 0, 0, 0);
                const uint32_t sum[4] = {(pb.x + ob.x) - (pa.x + oa.x), (pb.y + ob.y) - (pa.y + oa.y),
                                         (pb.z + ob.z) - (pa.z + oa.z), (pb.w + ob.w) - (pa.w + oa.w)};
                uint32_t wd[4];
                const uint32_t len = (uint32_t)(l + r + 1);
                if constexpr (PRIOR) {
                    // valid counts of the window from the count prefix (two 8-bit counts per word),
                    // validity from the centre pixel's range (the tile kernel's rule)
                    const uint2 cb = *reinterpret_cast<const uint2*>(s_cnt + b * W2 + k4);
                    const uint2 ca = a > 0 ? *reinterpret_cast<const uint2*>(s_cnt + (a - 1) * W2 + k4) : make_uint2(0, 0);
                    const uint2 tb = *reinterpret_cast<const uint2*>(s_totc + rhi * W2 + k4);
                    const uint2 ta = *reinterpret_cast<const uint2*>(s_totc + rlo * W2 + k4);
                    const uint32_t cw[4] = {(cb.x & 0xFFFFu) + (tb.x & 0xFFFFu) - (ca.x & 0xFFFFu) - (ta.x & 0xFFFFu),
                                            (cb.x >> 16) + (tb.x >> 16) - (ca.x >> 16) - (ta.x >> 16),
                                            (cb.y & 0xFFFFu) + (tb.y & 0xFFFFu) - (ca.y & 0xFFFFu) - (ta.y & 0xFFFFu),
                                            (cb.y >> 16) + (tb.y >> 16) - (ca.y >> 16) - (ta.y >> 16)};
                    const uint32_t rg = s_rng[sxi];
                    const int lo = (int)(int16_t)(rg & 0xFFFFu), hi = (int)(int16_t)(rg >> 16);
#pragma unroll
                    for (int q = 0; q < 4; ++q) wd[q] = prior_word<U8>(c, sum[q], cw[q] & 0xFFFFu, k4 + q, lo, hi, s_magic);
                } else if (2 * k4 + 8 <= c.D && len > 1 && x - l >= c.d0 + 2 * k4 + 7 && x + r <= c.w - 1 + c.d0 + 2 * k4) {
                    // these eight disparities have their whole window valid (inside the range, x - d inside
                    // the image over the window): one count, no per-word tests
                    const uint32_t mg = s_magic[len];
                    if constexpr (U8) {
                        // the quotients are the products' top bytes
                        uint32_t o[2];
#pragma unroll
                        for (int q = 0; q < 4; q += 2) {
                            const uint32_t e = __byte_perm((sum[q] & 0xFFFFu) * mg, (sum[q] >> 16) * mg, 0x0073);
                            const uint32_t f = __byte_perm((sum[q + 1] & 0xFFFFu) * mg, (sum[q + 1] >> 16) * mg, 0x0073);
                            o[q / 2] = __byte_perm(e, f, 0x5410);
                        }
                        *reinterpret_cast<uint2*>(reinterpret_cast<uint8_t*>(out_vol) + ((size_t)row + x) * (2 * W2) + 2 * k4) =
                            make_uint2(o[0], o[1]);
                        continue;
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        wd[q] = __byte_perm(__umulhi(sum[q] & 0xFFFFu, mg), __umulhi(sum[q] >> 16, mg), 0x5410);
                } else {
#pragma unroll
                    for (int q = 0; q < 4; ++q) wd[q] = agg_word<U8>(c, sum[q], k4 + q, x, l, r, s_magic);
                }
                if constexpr (U8)
                    *reinterpret_cast<uint2*>(reinterpret_cast<uint8_t*>(out_vol) + ((size_t)row + x) * (2 * W2) + 2 * k4) =
                        make_uint2(__byte_perm(wd[0], wd[1], 0x6420), __byte_perm(wd[2], wd[3], 0x6420));
                else
                    *reinterpret_cast<uint4*>(out_vol + ((size_t)row + x) * W2 + k4) = make_uint4(wd[0], wd[1], wd[2], wd[3]);
            }
        }
    }
}

// Shared memory one SM gives each of `per_sm` resident blocks.
size_t smem_per_block(int per_sm) {
    static size_t sm_total = 0, reserved = 0;
    if (!sm_total) {
        int dev = 0, v = 0, r = 0;
        if (cudaGetDevice(&dev) == cudaSuccess &&
            cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) == cudaSuccess &&
            cudaDeviceGetAttribute(&r, cudaDevAttrReservedSharedMemoryPerBlock, dev) == cudaSuccess) {
            sm_total = (size_t)v;
            reserved = (size_t)r;
        } else {
            cudaGetLastError();
            return 100 * 1024;
        }
    }
    return sm_total / per_sm - reserved;
}

// Tile width of the aggregating form: the fewest tiles per row (least halo) whose staging lets two
// 16-warp blocks share an SM (one block for 192 or 256 padded disparities); a requested width
// (tuning key cost_tile) wins when it fits one block.
int cross_tile(const CostCtx& c, int lmax, bool full) {
    const bool prior = c.prior_ranges != 0;
    if ((c.tile == 64 || c.tile == 128 || c.tile == 256) &&
        run_geom(c, c.tile, lmax, true, full, prior).total <= 200 * 1024)
        return c.tile;
    // one block per SM for the wide forms (see cost_run_kernel), else two
    const size_t budget = smem_per_block(c.Dp > 128 ? 1 : 2);
    for (int ntx = 1; ntx <= c.w; ++ntx) {
        const int txc = round_up((c.w + ntx - 1) / ntx, 4);
        // (with per-pixel ranges a warp's share of the output pixels is one a lane at most)
        if (prior && txc > 32 * run_warps(true)) continue;
        if (run_geom(c, txc, lmax, true, full, prior).total <= budget) return txc;
        if (txc <= 32) break;
    }
    return 32;
}

// Tile width without aggregation (no halo): eight runs of up to kMaxRun pixels.  A run's end costs its warp
// about kRunEnd steps more (the partial minima, the barrier), blocks walk the tiles in rounds whose last is
// partly empty, and warps past the row's end idle: the run length with the least rounds (half counted whole,
// half as the fraction used) times run, times the square of the padding.  Over run lengths of 20 to 120 at
// 640x480 to 1920x1080, D 64 to 256, the choice was within 9% of the best one (Fast 1920x1080 D256: 80 pixels
// 239 us, 32 pixels 276; 1280x720 D128: 80 pixels 67 us, 60 pixels 78).
constexpr int kMaxRun = 96, kRunEnd = 8;
int plain_tile(const CostCtx& c, int blocks) {
    const int nrun = run_warps(false);
    int best = 0;
    double best_cost = 0;
    for (int rl = 4; rl <= kMaxRun; rl += 4) {
        const int txc = rl * nrun, ntx = (c.w + txc - 1) / txc;
        const double rounds = (double)ntx * c.h / blocks, pad = (double)ntx * txc / c.w;
        const double cost = (std::ceil(rounds) + rounds) * (rl + kRunEnd) * pad * pad;
        if (!best || cost < best_cost) {
            best_cost = cost;
            best = txc;
        }
    }
    return best;
}

template <bool CROSS, bool STORE, bool FULL, int WPL, bool PRIOR, bool U8>
cudaError_t launch_runs_w(const CostCtx& c, int txc, int lmax, int tau, uint32_t* vol, uint32_t* rkey,
                          const uint32_t* magic, cudaStream_t s) {
    RunGeom g = run_geom(c, txc, CROSS ? lmax : 0, CROSS, FULL, PRIOR);
    const int nt = 32 * g.nrun;
    auto kern = cost_run_kernel<CROSS, STORE, FULL, WPL, PRIOR, U8>;
    cudaError_t e = allow_dynamic_smem(kern, g.total);
    if (e != cudaSuccess) return e;
    int per_sm = 0, dev = 0, nsm = 0;
    e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, nt, g.total);
    if (e != cudaSuccess) return e;
    // the widest tile's staging decided the occupancy; a narrower one needs less
    if (!CROSS) g = run_geom(c, plain_tile(c, std::max(1, per_sm) * nsm), 0, CROSS, FULL, PRIOR);
    const int blocks = std::max(1, std::min(g.ntiles, std::max(1, per_sm) * nsm));
    kern<<<blocks, nt, g.total, s>>>(c, g, lmax, tau, vol, rkey, magic);
    return cudaGetLastError();
}

// Words per lane as a compile-time constant: one warp spans Dp = 64 * WPL disparities.
template <bool CROSS, bool STORE, bool FULL, bool PRIOR>
cudaError_t launch_runs_p(const CostCtx& c, int txc, int lmax, int tau, uint32_t* vol, uint32_t* rkey,
                          const uint32_t* magic, cudaStream_t s) {
    if constexpr (STORE && (CROSS || !FULL)) {
        // the byte volume (costs below 255): census-only, or aggregated
        if (c.vol8) {
            switch (c.Dp) {
                case 64: return launch_runs_w<CROSS, STORE, FULL, 1, PRIOR, true>(c, txc, lmax, tau, vol, rkey, magic, s);
                case 128: return launch_runs_w<CROSS, STORE, FULL, 2, PRIOR, true>(c, txc, lmax, tau, vol, rkey, magic, s);
                case 192: return launch_runs_w<CROSS, STORE, FULL, 3, PRIOR, true>(c, txc, lmax, tau, vol, rkey, magic, s);
                default: return launch_runs_w<CROSS, STORE, FULL, 4, PRIOR, true>(c, txc, lmax, tau, vol, rkey, magic, s);
            }
        }
    } else {
        if (c.vol8) return cudaErrorInvalidValue;
    }
    switch (c.Dp) {
        case 64: return launch_runs_w<CROSS, STORE, FULL, 1, PRIOR, false>(c, txc, lmax, tau, vol, rkey, magic, s);
        case 128: return launch_runs_w<CROSS, STORE, FULL, 2, PRIOR, false>(c, txc, lmax, tau, vol, rkey, magic, s);
        case 192: return launch_runs_w<CROSS, STORE, FULL, 3, PRIOR, false>(c, txc, lmax, tau, vol, rkey, magic, s);
        default: return launch_runs_w<CROSS, STORE, FULL, 4, PRIOR, false>(c, txc, lmax, tau, vol, rkey, magic, s);
    }
}

template <bool CROSS, bool STORE, bool FULL>
cudaError_t launch_runs_t(const CostCtx& c, int txc, int lmax, int tau, uint32_t* vol, uint32_t* rkey,
                          const uint32_t* magic, cudaStream_t s) {
    if (c.prior_ranges) return launch_runs_p<CROSS, STORE, FULL, true>(c, txc, lmax, tau, vol, rkey, magic, s);
    return launch_runs_p<CROSS, STORE, FULL, false>(c, txc, lmax, tau, vol, rkey, magic, s);
}

}  // namespace

size_t cost_runs_smem_bytes(const CostCtx& c, int mode, int lmax) {
    const bool full = c.use_ad || c.use_grad;
    const bool prior = c.prior_ranges != 0;
    if (mode == 1) return run_geom(c, cross_tile(c, lmax, full), lmax, true, full, prior).total;
    return run_geom(c, kMaxRun * run_warps(false), 0, false, full, prior).total;
}

bool cost_runs_supported(const CostCtx& c, int mode, int lmax) {
    if (c.kernel == 1 || c.census64) return false;
    if (c.Dp % 64 != 0 || c.Dp > 256) return false;
    const bool full = c.use_ad || c.use_grad;
    if (mode == 2 && (full || c.prior_ranges)) return false;  // the fused form: census-only, default ranges
    if (mode == 1 && lmax > 127) return false;
    // the staging must fit the per-block budget the tile width was chosen for
    return cost_runs_smem_bytes(c, mode, lmax) <= smem_per_block(c.Dp > 128 && mode == 1 ? 1 : 2);
}

cudaError_t launch_cost_runs(const CostCtx& c, int mode, int lmax, int tau, uint32_t* vol, uint32_t* rkey,
                             const uint32_t* magic, cudaStream_t s) {
    const bool full = c.use_ad || c.use_grad;
    if (mode == 1) {
        const int txc = cross_tile(c, lmax, full);
        return full ? launch_runs_t<true, true, true>(c, txc, lmax, tau, vol, rkey, magic, s)
                    : launch_runs_t<true, true, false>(c, txc, lmax, tau, vol, rkey, magic, s);
    }
    if (mode == 0)
        return full ? launch_runs_t<false, true, true>(c, kMaxRun * run_warps(false), lmax, tau, vol, rkey, magic, s)
                    : launch_runs_t<false, true, false>(c, kMaxRun * run_warps(false), lmax, tau, vol, rkey, magic, s);
    return launch_runs_t<false, false, false>(c, kMaxRun * run_warps(false), lmax, tau, vol, rkey, magic, s);
}

}  // namespace apgcu
