// Vertical half of the Cross-arm aggregation over byte volumes, CostAggregator::aggregate_hv
// (src/cost_aggregator.cpp:107-138): T(x, y, d), the horizontally aggregated costs, and the result at one
// byte per voxel (0xFF invalid), for configurations whose quantised costs stay below 255 and arms of at
// most kMaxArm pixels (every preset).  Results are those of cross.cu's kernels.
//
// A thread owns eight consecutive disparities of one pixel column and slides down a segment of rows.  The
// column's prefix sums (two disparities to a 32-bit word, four words) of the live rows lie in a
// shared-memory ring; an output row is the difference of two ring entries, a multiply by the window
// length's reciprocal and a byte pack:
//   * the prefix words hold the even and the odd disparities of four bytes, so widening a row's bytes is
//     one and / one permute a word, and a 32-bit difference of two prefixes is exact in both halves (a
//     window's low halves sum to less than 2^16; see cross.cu);
//   * floor(s / n) for s <= 254 n is the top byte of the 32-bit product s * m, m = floor(2^24 / n) + 1:
//     s * m = 2^24 s / n + s e / n with e <= n, and s e < 2^24 for n <= 255, so the floor is exact, and
//     s * m <= 254 (2^24 + n) < 2^32.  The quotients are packed by byte permutes with no shift or mask;
//   * arms, ring offsets and the reciprocal are computed once per pixel and shared by its threads.
// COUNT (per-pixel ranges, negative disparities): the window count varies with the disparity, so a second
// ring keeps prefix sums of the valid flags (a byte per disparity: at most 2 kMaxArm + 1 per window), each
// disparity looks its reciprocal up by its own count, and the centre pixel's range masks the result.
//
// Bound: the integer pipes, about 55 instructions per row of eight disparities (the 16-bit form took
// about five times the instructions per voxel).
#include "common.cuh"
#include "kernels.h"

#include <algorithm>
#include <type_traits>

namespace apgcu {

namespace {

constexpr int kMaxArm = 17;
constexpr int kRows = 4;                         // output rows (and rows pushed) per chunk
constexpr int kSlots = 2 * kMaxArm + 2 * kRows;  // live prefixes: rows y - arm - 1 .. y + arm + 2 kRows - 2
constexpr int kAhead = 4;                        // chunks of rows in flight

// Per pixel of the block's segment: byte offsets of the window's ends from the row's ring slot
// (down * stride | (up + 1) * stride << 16) and the reciprocal of its length.
struct PixelWin {
    uint32_t off, mul;
};

__device__ __forceinline__ uint32_t shl_clamp(uint32_t v, uint32_t n) {
    uint32_t r;
    asm("shl.b32 %0, %1, %2;" : "=r"(r) : "r"(v), "r"(n));  // 0 for n >= 32
    return r;
}
// Bytes [a, b) of a four-byte word.
__device__ __forceinline__ uint32_t byte_span(int a, int b) {
    return (shl_clamp(1u, 8u * (uint32_t)max(b, 0)) - 1u) & ~(shl_clamp(1u, 8u * (uint32_t)max(a, 0)) - 1u);
}

// NT threads with disparities per block at most; tpc = Dp / 8 of them per column.
template <bool COUNT, int NT>
__global__ void __launch_bounds__(NT) cross_v8_kernel(int w, int h, int d0, int D, int Dp, int lmax, int tau, int cols,
                                                      int seg, const uint8_t* __restrict__ gray,
                                                      const int16_t* __restrict__ rmin,
                                                      const int16_t* __restrict__ rmax,
                                                      const uint8_t* __restrict__ tin, uint8_t* __restrict__ cout) {
    constexpr uint32_t STRIDE = NT * 16, RING = kSlots * STRIDE;  // bytes
    extern __shared__ __align__(16) unsigned char smem[];
    uint32_t* s_mul = reinterpret_cast<uint32_t*>(smem + RING + (COUNT ? RING / 2 : 0));  // reciprocal by count
    PixelWin* s_win = reinterpret_cast<PixelWin*>(s_mul + 2 * kMaxArm + 2);                 // [seg][cols]
    uint32_t* s_rng = reinterpret_cast<uint32_t*>(s_win + seg * cols);                      // [seg][cols] (COUNT)
    uint32_t* s_gray = s_rng + (COUNT ? seg * cols : 0);  // [seg + 2 lmax][gw] words of four columns
    const int xb = blockIdx.x * cols, y0 = blockIdx.y * seg, y1 = min(h, y0 + seg);
    const int tid = threadIdx.x;
    const int gs = y1 - y0 + 2 * lmax, gw = (cols + 3) / 4;

    for (int i = tid; i < 2 * kMaxArm + 2; i += NT) s_mul[i] = i ? (1u << 24) / (uint32_t)i + 1u : 0u;
    for (int i = tid; i < gs * gw * 4; i += NT) {
        const int r = i / (gw * 4), cc = i - r * (gw * 4);
        const int yy = y0 - lmax + r, x = xb + cc;
        reinterpret_cast<uint8_t*>(s_gray)[i] = (cc < cols && x < w && yy >= 0 && yy < h) ? gray[yy * w + x] : 0;
    }
    __syncthreads();
    // arms (build_cross_arms, src/cost_aggregator.cpp:17-63), four columns at a time: a byte's run lasts
    // while its difference from the centre stays within tau, and ends at the image's border.  A byte
    // exceeds tau when its top bit is set in (d & 0x7F) + (0x7F - tau) or in d itself (tau below 128), or
    // in both (tau - 128 in place of tau).
    const int tc = min(tau, 255);
    const uint32_t kadd = (uint32_t)(0x7F - (tc & 0x7F)) * 0x01010101u;
    for (int i = tid; i < (y1 - y0) * gw; i += NT) {
        const int r = i / gw, c4 = i - r * gw, yy = y0 + r;
        const uint32_t* g = s_gray + (r + lmax) * gw + c4;
        const uint32_t c0 = g[0];
        uint32_t run[2];
#pragma unroll
        for (int dir = 0; dir < 2; ++dir) {
            uint32_t alive = tau >= 0 ? 0x01010101u : 0u, n = 0;
            for (int k = 1; k <= lmax && alive; ++k) {
                const uint32_t d = __vabsdiffu4(dir ? g[k * gw] : g[-k * gw], c0);
                const uint32_t t = (d & 0x7F7F7F7Fu) + kadd;
                alive &= ~((tc < 128 ? t | d : t & d) >> 7);
                n += alive;
            }
            run[dir] = n;
        }
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int cc = 4 * c4 + b, x = xb + cc;
            if (cc >= cols) break;
            const int u = min((int)((run[0] >> (8 * b)) & 0xFFu), yy);
            const int v = min((int)((run[1] >> (8 * b)) & 0xFFu), h - 1 - yy);
            s_win[r * cols + cc] = PixelWin{(uint32_t)v * STRIDE | ((uint32_t)(u + 1) * STRIDE << 16), s_mul[u + v + 1]};
            if (COUNT)
                s_rng[r * cols + cc] =
                    x < w ? (uint32_t)(uint16_t)rmin[yy * w + x] | ((uint32_t)(uint16_t)rmax[yy * w + x] << 16) : 0u;
        }
    }
    __syncthreads();
    const int tpc = Dp / 8;
    const int ci = tid / tpc, j = tid - ci * tpc;
    const int x = xb + ci;
    if (ci >= cols || x >= w) return;

    // default ranges: disparities past x or the range are invalid in every row of the column
    uint32_t inv0 = 0, inv1 = 0;
    if (!COUNT) {
        const int nv = min(D, x - d0 + 1) - 8 * j;  // valid disparities of this thread
        inv0 = ~byte_span(0, min(nv, 4));
        inv1 = ~byte_span(0, min(nv - 4, 4));
    }
    const int ystart = max(0, y0 - lmax), yend = min(h, y1 + lmax);  // rows read
    unsigned char* ring = smem;
    unsigned char* ringc = smem + RING;
    const uint32_t me = (uint32_t)tid * 16;
    *reinterpret_cast<uint4*>(ring + me) = make_uint4(0, 0, 0, 0);  // the prefix before row ystart
    if (COUNT) *reinterpret_cast<uint2*>(ringc + me / 2) = make_uint2(0, 0);

    const size_t rowb = (size_t)w * Dp;
    const uint8_t* src = tin + ((size_t)ystart * w + x) * Dp + 8 * j;  // the next row to load
    uint8_t* dst = cout + ((size_t)y0 * w + x) * Dp + 8 * j;           // row y
    int loaded = ystart, pushed = ystart;
    uint4 ps = make_uint4(0, 0, 0, 0);
    uint2 pc = make_uint2(0, 0);
    uint32_t pslot = STRIDE + me;                                           // slot of row `pushed`
    uint32_t yslot = (uint32_t)((y0 - ystart + 1) % kSlots) * STRIDE + me;  // slot of row y
    // rows past yend load as zeros and are pushed into slots nothing reads
    auto load = [&](uint2 (&q)[kRows]) {
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
            q[i] = make_uint2(0, 0);
            if (loaded + i < yend) q[i] = __ldcs(reinterpret_cast<const uint2*>(src + i * rowb));
        }
        loaded += kRows;
        src += kRows * rowb;
    };
    auto push = [&](const uint2 (&q)[kRows]) {
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
            uint32_t a = q[i].x, b = q[i].y;
            if constexpr (COUNT) {
                const uint32_t ia = (((a & 0x7F7F7F7Fu) + 0x01010101u) & a & 0x80808080u) >> 7;  // 1 where 0xFF
                const uint32_t ib = (((b & 0x7F7F7F7Fu) + 0x01010101u) & b & 0x80808080u) >> 7;
                a -= ia * 255u;
                b -= ib * 255u;
                pc.x += ia ^ 0x01010101u;
                pc.y += ib ^ 0x01010101u;
                *reinterpret_cast<uint2*>(ringc + pslot / 2) = pc;
            }
            ps.x += a & 0x00FF00FFu;
            ps.y += __byte_perm(a, 0u, 0x4341);
            ps.z += b & 0x00FF00FFu;
            ps.w += __byte_perm(b, 0u, 0x4341);
            *reinterpret_cast<uint4*>(ring + pslot) = ps;
            pslot += STRIDE;
            pslot = min(pslot, pslot - RING);  // unsigned: wraps past the ring's end
        }
        pushed += kRows;
    };
    // N output rows from row y: the rows' windows first, then every ring read, then the quotients
    auto emit = [&](auto nt, int y) {
        constexpr int N = decltype(nt)::value;
        uint4 sb[N], sa[N];
        uint2 cb[COUNT ? N : 1], ca[COUNT ? N : 1];
        uint32_t mul[N];
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const PixelWin wn = s_win[(y + i - y0) * cols + ci];
            uint32_t ob = yslot + (wn.off & 0xFFFFu), oa = yslot - (wn.off >> 16);
            ob = min(ob, ob - RING);
            oa = min(oa, oa + RING);
            yslot += STRIDE;
            yslot = min(yslot, yslot - RING);
            sb[i] = *reinterpret_cast<const uint4*>(ring + ob);
            sa[i] = *reinterpret_cast<const uint4*>(ring + oa);
            mul[i] = wn.mul;
            if constexpr (COUNT) {
                cb[i] = *reinterpret_cast<const uint2*>(ringc + ob / 2);
                ca[i] = *reinterpret_cast<const uint2*>(ringc + oa / 2);
            }
        }
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const uint32_t s[4] = {sb[i].x - sa[i].x, sb[i].y - sa[i].y, sb[i].z - sa[i].z, sb[i].w - sa[i].w};
            uint32_t o[2];
            if constexpr (!COUNT) {
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const uint32_t e = s[2 * k], f = s[2 * k + 1];  // even, odd disparities
                    const uint32_t p0 = (e & 0xFFFFu) * mul[i], p2 = (e >> 16) * mul[i];
                    const uint32_t p1 = (f & 0xFFFFu) * mul[i], p3 = (f >> 16) * mul[i];
                    o[k] = __byte_perm(__byte_perm(p0, p1, 0x0073), __byte_perm(p2, p3, 0x0073), 0x5410);
                }
                o[0] |= inv0;
                o[1] |= inv1;
            } else {
                const uint32_t n[2] = {cb[i].x - ca[i].x, cb[i].y - ca[i].y};
                const uint32_t rg = s_rng[(y + i - y0) * cols + ci];
                const int lo = (int)(int16_t)(rg & 0xFFFFu) - d0 - 8 * j;
                const int hi = min((int)(int16_t)(rg >> 16) - d0, D) - 8 * j;
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const uint32_t e = s[2 * k], f = s[2 * k + 1], c = n[k];
                    const uint32_t p0 = (e & 0xFFFFu) * s_mul[c & 0xFFu], p2 = (e >> 16) * s_mul[(c >> 16) & 0xFFu];
                    const uint32_t p1 = (f & 0xFFFFu) * s_mul[(c >> 8) & 0xFFu], p3 = (f >> 16) * s_mul[c >> 24];
                    o[k] = __byte_perm(__byte_perm(p0, p1, 0x0073), __byte_perm(p2, p3, 0x0073), 0x5410);
                    // invalid: no valid voxel in the window (counts are below 0x80), or outside the range
                    const uint32_t zero = (~(c + 0x7F7F7F7Fu) & 0x80808080u) >> 7;
                    o[k] |= zero * 255u | ~byte_span(min(lo - 4 * k, 4), min(hi - 4 * k, 4));
                }
            }
            __stcs(reinterpret_cast<uint2*>(dst), make_uint2(o[0], o[1]));
            dst += rowb;
        }
    };
    auto emit_chunk = [&](int y) {
        if (y + kRows <= y1) {
            emit(std::integral_constant<int, kRows>(), y);
        } else {
            for (int i = y; i < y1; ++i) emit(std::integral_constant<int, 1>(), i);
        }
    };
    // kAhead chunks of rows in flight.  Before the first output they move up through the buffers; then the
    // buffers are pushed in turn, so that no register move waits for a load just issued
    uint2 q[kAhead][kRows];
#pragma unroll
    for (int k = 0; k < kAhead; ++k) load(q[k]);
    for (int first = min(yend, min(y0 + kRows, y1) + lmax) - ystart; pushed - ystart < first;) {
        push(q[0]);
#pragma unroll
        for (int k = 0; k + 1 < kAhead; ++k)
#pragma unroll
            for (int i = 0; i < kRows; ++i) q[k][i] = q[k + 1][i];
        load(q[kAhead - 1]);
    }
    for (int y = y0; y < y1; y += kAhead * kRows) {
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
            if (y + k * kRows < y1) emit_chunk(y + k * kRows);
            push(q[k]);
            load(q[k]);
        }
    }
}

template <bool COUNT, int NT>
cudaError_t launch_t(int w, int h, int d0, int D, int Dp, int lmax, int tau, const uint8_t* gray, const int16_t* rmin,
                     const int16_t* rmax, const uint8_t* tin, uint8_t* cout, cudaStream_t s) {
    const int cols = std::max(1, NT / (Dp / 8));
    auto kern = cross_v8_kernel<COUNT, NT>;
    auto bytes = [&](int seg) {
        return (size_t)kSlots * NT * (COUNT ? 24 : 16) + (2 * kMaxArm + 2) * 4 + (size_t)seg * cols * (COUNT ? 12 : 8) +
               (size_t)(seg + 2 * lmax) * ((cols + 3) / 4) * 4;
    };
    // segments of rows: tall ones re-read fewer halo rows (2 lmax each, plus a prologue worth about kFixed
    // rows), short ones fill the device's last wave; the count of the least waves x rows
    int dev = 0, nsm = 148, per_sm = 228 * 1024, reserved = 1024;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev) != cudaSuccess)
        cudaGetLastError();
    constexpr int kFixed = 24;
    const int nbx = (w + cols - 1) / cols;
    int seg = 16;
    long long best = -1;
    for (int ns = 1; ns <= (h + 15) / 16; ++ns) {
        const int sg = (h + ns - 1) / ns;
        const int fit = per_sm / (int)(bytes(sg) + reserved);
        if (fit < 1 || (long long)bytes(sg) > per_sm - reserved) continue;
        // blocks of an SM share its issue slots: a wave of `fit` blocks takes as long as fit blocks' rows
        const long long waves = ((long long)nbx * ns + (long long)nsm * fit - 1) / ((long long)nsm * fit);
        const long long cost = waves * (2 + fit) * (sg + 2 * lmax + kFixed);
        if (best < 0 || cost < best) {
            best = cost;
            seg = sg;
        }
    }
    const cudaError_t e = allow_dynamic_smem(kern, bytes(seg));
    if (e != cudaSuccess) return e;
    dim3 grid((w + cols - 1) / cols, (h + seg - 1) / seg);
    kern<<<grid, NT, bytes(seg), s>>>(w, h, d0, D, Dp, lmax, tau, cols, seg, gray, rmin, rmax, tin, cout);
    return cudaGetLastError();
}

}  // namespace

bool cross_v8_supported(int Dp, int lmax) { return Dp <= 256 && Dp % 64 == 0 && lmax <= kMaxArm; }

cudaError_t launch_cross_v8(int w, int h, int d0, int D, int Dp, int lmax, int tau, const uint8_t* gray,
                            const int16_t* rmin, const int16_t* rmax, const uint8_t* tin, uint8_t* cout,
                            bool default_ranges, cudaStream_t s) {
    if (!cross_v8_supported(Dp, lmax)) return cudaErrorInvalidValue;
    // 128 threads: two blocks of a sum ring on an SM; 64 threads: three of a sum and a count ring
    if (default_ranges && d0 >= 0) return launch_t<false, 128>(w, h, d0, D, Dp, lmax, tau, gray, rmin, rmax, tin, cout, s);
    return launch_t<true, 64>(w, h, d0, D, Dp, lmax, tau, gray, rmin, rmax, tin, cout, s);
}

}  // namespace apgcu
