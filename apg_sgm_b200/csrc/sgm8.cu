// Semi-global matching sweeps over the byte volume, two scanlines per warp.
//
// Restates the recurrence of sgm.cu (SgmOptimizer::process_pixel, src/sgm_optimizer.cpp:44-80, and
// wta_impl, :436-555) for configurations whose quantised costs stay below 255 and whose largest P2
// is at most 255 (every preset), at up to 256 padded disparities:
//   * the volume holds one byte per voxel (0xFF invalid);
//   * with the path value L(d) = C(d) + delta(d), delta(d) = min(L'(d), L'(d-1) + P1, L'(d+1) + P1,
//     m' + P2) - m' lies in [0, P2].  The sweeps of the first phase store delta, one byte per voxel
//     and direction, instead of the 16-bit path value; the sum over n directions is n * C + the sum
//     of the deltas, exactly.  The sums leave the device only through the WTA (and stage dumps).
//     Per voxel the first phase moves 2 bytes a direction where 16-bit path values over a 16-bit
//     volume took 4, the last sweep 1 + (n - 1) where it took 2 n, and eight directions need no fold;
//   * a warp runs two neighbouring scanlines of one direction: a 32-bit word holds the path values
//     of one disparity, scanline A's in the low half and scanline B's in the high half.  Neighbouring
//     disparities are neighbouring words, so the recurrence needs no byte permutes and one shuffle
//     each way serves both scanlines; widening bytes to halves costs 1.5 operations a word, which
//     interleaves the scanlines at the same time;
//   * per word: t = min(L'(d-1), L'(d+1)); x = min(t + P1, L'(d)); delta = min(x - m', P2);
//     L = C + delta: three DPX / SIMD minima and one 32-bit add.  m' enters last, so the warp's two
//     min-reductions run beside the neighbour shuffles and the first two minima.
// Values (each biased by 0x0400): valid costs are at most 254 and valid path values at most 254 + 255 = 509.
// An invalid cost is widened to 0x03FF, a padded one to at least 0x0300 = 768.  The room is tight: no valid
// entry takes a candidate from an invalid neighbour while 768 > m' + P2 for every valid m', so 768 - 509 = 259
// must exceed the largest P2, 255.  All halves of path values stay below 0x2000, so plain 32-bit adds never
// carry between them and the signed minima are exact.  A pixel whose predecessor has no valid entry (m' >=
// 0x0300) takes L = C: P2 reads as 0 there, which makes every delta 0; the first pixel of a scanline does the
// same with L' = 0.
//
// Steps whose pixels have every disparity of the range valid (default ranges: x >= dmax - 1) skip the
// invalid-byte test: only the padded disparities are invalid there, a constant mask per lane.
//
// Loads run one to three groups of steps ahead through a per-warp shared-memory ring, a cp.async group each,
// 16 bytes per lane: at 256 padded disparities one copy instruction brings both scanlines' costs of a step, at
// 64 those of four.  Bound: HBM for full frames (1920x1080 D256: the first phase at 91% of the copy rate, the
// last sweep at 76%), else each step's dependent chain (reduction, two minima, add; 135 cycles at 640x480
// D64).
#include "sgm8.cuh"

#include <algorithm>
#include <cstddef>
#include <cstring>
#include <vector>

namespace apgcu {

namespace {

constexpr int kMaxIn = 7;                   // first-phase directions of Path8
// Halves of a path-value word: kBias + L.  The bias keeps a low half above zero, so that one 32-bit
// subtraction negates both halves (n = 0x10000 - acc, exact in each half modulo 2^16).
constexpr uint32_t kBias = 0x0400u;
constexpr uint32_t kBias2 = 0x04000400u;
constexpr uint32_t kInvalid = 0x0300u;      // invalid path values are at least this, valid ones below
constexpr uint32_t kPad2 = 0x07000700u;     // bias and the invalid marker (with the byte 0xFF: 0x03FF)
constexpr uint32_t kEdge2 = 0x0FFF0FFFu;    // beyond the ends of the range: above every path value
// A max-reduction of negated minima holds -(kBias + m') in its high half; below this m' is invalid.
constexpr uint32_t kNoPred = (0x10000u - kBias - kInvalid) << 16;
constexpr uint32_t kFresh = (0x10000u - kBias) << 16;  // m' = 0
constexpr uint32_t kMaxCost = 254, kMaxP2 = 255;       // what the callers keep to (sgm8_supported, the engine's layout)
static_assert(kPad2 == (kBias + kInvalid) * 0x00010001u, "padded disparities are invalid");
static_assert(kInvalid > kMaxCost + kMaxP2 + kMaxP2, "an invalid neighbour never wins over m' + P2");
static_assert((kEdge2 & 0xFFFFu) > kBias + (kInvalid | 0xFFu) + kMaxP2 + kMaxP2, "nor does the edge");
static_assert((kBias + (kInvalid | 0xFFu) + kMaxP2) * (kMaxIn + 1) < 0x8000u, "sums of all directions fit their halves");

struct Args8 {
    int w, h, d0, D, dmax;
    int def_ranges;  // every pixel has the default range
    int P1;
    alignas(16) uint8_t p2[256];  // adaptive P2 by |gray difference|
    const uint8_t* gray;
    const uint8_t* vol;
    WtaOut wta;
    uint32_t* sum;  // final sums (u16, 0xFFFF invalid) for stage dumps, or null
    int t_begin, t_end;
    uint32_t* carry;
};
static_assert(offsetof(Args8, p2) % 8 == 0, "gray_init copies the table eight bytes a lane");
struct Dirs8 {
    int n;
    int dx[kMaxIn], dy[kMaxIn], nscan[kMaxIn];
    int warp_begin[kMaxIn + 1];
    uint8_t* out[kMaxIn];
};
struct In8 {
    const uint8_t* d[kMaxIn];
};

// W disparities per lane, AL lanes with disparities, CH 16-byte chunks per pixel.
template <int DP>
struct Geo {
    static constexpr int W = DP == 64 ? 2 : (DP == 128 ? 4 : 8);
    static constexpr int AL = DP / W;
    static constexpr int CH = DP / 16;
    static constexpr int SPI = 32 / (2 * CH);  // steps (both scanlines) per 16-byte copy instruction
    static constexpr int RS = DP / 2 + 4;  // words per row of the WTA buffer: 4 mod 32, so 16-byte accesses
                                           // of eight rows fall in distinct banks
    static constexpr int wta_words = 32 * RS;
};
constexpr int kTail = 64;  // bytes behind a ring: idle lanes (192 padded disparities) read past a slot

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) { return __byte_perm(a, b, sel); }

__device__ __forceinline__ void cp16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// This lane's words of one pixel of both scanlines (A's slice at a, B's DP bytes on).
template <int DP>
struct Raw {
    static constexpr int N = Geo<DP>::W >= 8 ? 2 : 1;
    uint32_t a[N], b[N];
};
template <int DP>
__device__ __forceinline__ Raw<DP> load_raw(const uint8_t* p) {
    Raw<DP> r;
    if constexpr (Geo<DP>::W == 2) {
        r.a[0] = *reinterpret_cast<const uint16_t*>(p);
        r.b[0] = *reinterpret_cast<const uint16_t*>(p + DP);
    } else if constexpr (Geo<DP>::W == 4) {
        r.a[0] = *reinterpret_cast<const uint32_t*>(p);
        r.b[0] = *reinterpret_cast<const uint32_t*>(p + DP);
    } else {
        const uint2 va = *reinterpret_cast<const uint2*>(p), vb = *reinterpret_cast<const uint2*>(p + DP);
        r.a[0] = va.x; r.a[1] = va.y;
        r.b[0] = vb.x; r.b[1] = vb.y;
    }
    return r;
}
// u[i]: bytes 2i, 2i + 1 of scanline A, then of scanline B.
template <int DP>
__device__ __forceinline__ void interleave(const Raw<DP>& r, uint32_t (&u)[Geo<DP>::W / 2]) {
    u[0] = prmt(r.a[0], r.b[0], 0x5410);
    if constexpr (Geo<DP>::W >= 4) u[1] = prmt(r.a[0], r.b[0], 0x7632);
    if constexpr (Geo<DP>::W == 8) {
        u[2] = prmt(r.a[1], r.b[1], 0x5410);
        u[3] = prmt(r.a[1], r.b[1], 0x7632);
    }
}

// State of a warp's two chains: path values, the neighbouring lanes' words (shuffled as soon as a step
// has its values, so the shuffles and the reductions run under the next step's loads), and the
// reductions' results: -(kBias + m') in the high halves of lo (A) and hi (B).
template <int W>
struct Chain {
    uint32_t L[W];
    uint32_t q[W];  // L + P1
    uint32_t up, dn, lo, hi;
};

template <int W>
__device__ __forceinline__ void chain_reduce(Chain<W>& s) {
    s.up = __shfl_up_sync(0xffffffffu, s.q[W - 1], 1);
    s.dn = __shfl_down_sync(0xffffffffu, s.q[0], 1);
    uint32_t acc = s.L[0];
#pragma unroll
    for (int k = 1; k + 1 < W; k += 2) acc = __vimin3_s16x2(acc, s.L[k], s.L[k + 1]);
    acc = __vmins2(acc, s.L[W - 1]);
    const uint32_t n = 0x00010000u - acc;
    s.lo = __reduce_max_sync(0xffffffffu, n << 16);
    s.hi = __reduce_max_sync(0xffffffffu, n);
}
template <int W>
__device__ __forceinline__ void chain_init(Chain<W>& s) {
#pragma unroll
    for (int k = 0; k < W; ++k) s.L[k] = s.q[k] = kBias2;
    s.up = s.dn = kBias2;
    s.lo = s.hi = kFresh;
}

// One step of both chains: r (the volume's bytes), p2 (A | B << 16) -> the deltas.  pad[k]: kPad2 for
// words past the range, else kBias2.  c receives the widened, biased costs.
template <int DP, bool CLEAN>
__device__ __forceinline__ void path_step(Chain<Geo<DP>::W>& s, const Raw<DP>& r, const uint32_t (&pad)[Geo<DP>::W],
                                          uint32_t p1x2, uint32_t p2, int lane, uint32_t (&c)[Geo<DP>::W],
                                          uint32_t (&dl)[Geo<DP>::W]) {
    constexpr int W = Geo<DP>::W;
    uint32_t u[W / 2];
    interleave<DP>(r, u);
#pragma unroll
    for (int i = 0; i < W / 2; ++i) {
        c[2 * i] = (u[i] & 0x00FF00FFu) | pad[2 * i];
        c[2 * i + 1] = prmt(u[i], pad[2 * i + 1], 0x7351);
    }
    if constexpr (!CLEAN) {
#pragma unroll
        for (int k = 0; k < W; ++k) {
            const uint32_t inv = (c[k] + 0x00010001u) & 0x01000100u;  // 0x100 where the byte is 0xFF
            c[k] += inv * 3u;                                          // 0xFF -> 0x03FF
        }
        p2 &= (s.lo > kNoPred ? 0x0000FFFFu : 0u) | (s.hi > kNoPred ? 0xFFFF0000u : 0u);
    }
    const uint32_t up = lane == 0 ? kEdge2 : s.up;
    const uint32_t dn = lane == Geo<DP>::AL - 1 ? kEdge2 : s.dn;
    const uint32_t nm = prmt(s.lo, s.hi, 0x7632);
#pragma unroll
    for (int k = 0; k < W; ++k) {
        const uint32_t x = __vimin3_s16x2(k == 0 ? up : s.q[k - 1], k == W - 1 ? dn : s.q[k + 1], s.L[k]);
        dl[k] = __viaddmin_s16x2(x, nm, p2);
    }
#pragma unroll
    for (int k = 0; k < W; ++k) {
        s.L[k] = c[k] + dl[k];
        s.q[k] = s.L[k] + p1x2;
    }
    chain_reduce(s);
}

// First pixel and length of scanline s (0 when s is past the last one).
__device__ __forceinline__ void scan_start8(int w, int h, int dx, int dy, int s, int nscan, int& x, int& y, int& len) {
    x = 0; y = 0; len = 0;
    if (s >= nscan) return;
    if (dy == 0) {
        y = s; x = dx > 0 ? 0 : w - 1; len = w;
    } else if (dx == 0) {
        x = s; y = dy > 0 ? 0 : h - 1; len = h;
    } else {
        // ray s: start pixel whose predecessor (x - dx, y - dy) is outside the image (the reference's
        // ray enumeration, src/sgm_optimizer.cpp:325-365)
        if (s < w) { x = s; y = dy > 0 ? 0 : h - 1; }
        else { x = dx > 0 ? 0 : w - 1; y = dy > 0 ? (s - w + 1) : (h - 1 - (s - w + 1)); }
        const int rx = dx > 0 ? w - x : x + 1;
        const int ry = dy > 0 ? h - y : y + 1;
        len = rx < ry ? rx : ry;
    }
}

// The geometry of a warp's two scanlines.
struct Pair {
    int xA, pA, lenA, xB, pB, lenB, step, maxlen, minlen;
    int fullA, fullB;  // the scanlines' own lengths (a band cuts the others)
};
__device__ __forceinline__ Pair pair_start(const Args8& a, int dx, int dy, int s, int nscan) {
    Pair q;
    int y;
    scan_start8(a.w, a.h, dx, dy, s, nscan, q.xA, y, q.lenA);
    q.pA = y * a.w + q.xA;
    // an odd last scanline runs as both halves of its warp (the same values, stored twice; pB == pA)
    scan_start8(a.w, a.h, dx, dy, s + 1 < nscan ? s + 1 : s, nscan, q.xB, y, q.lenB);
    q.pB = y * a.w + q.xB;
    q.step = dy * a.w + dx;
    q.maxlen = max(q.lenA, q.lenB);
    q.minlen = min(q.lenA, q.lenB);
    q.fullA = q.lenA;
    q.fullB = q.lenB;
    return q;
}
// P2 of a warp's steps, 32 at a time: lane j looks up step t0 + j of both scanlines (the grays prefetched
// one block ahead, through clamped addresses: a select behind a load would wait for it) and leaves
// P2(A) | P2(B) << 16 in shared memory, from where a group of steps reads its words together.
struct P2Smem {
    uint32_t w[32];
    uint8_t lut[256];
};
struct GrayRun {
    int nextA, nextB, carryA, carryB;
};
__device__ __forceinline__ void gray_load(const Args8& a, const Pair& q, int t, GrayRun& g) {
    g.nextA = (int)__ldg(a.gray + q.pA + min(t, q.fullA - 1) * q.step);
    g.nextB = (int)__ldg(a.gray + q.pB + min(t, q.fullB - 1) * q.step);
}
__device__ __forceinline__ void gray_init(const Args8& a, const Pair& q, int tb, int lane, P2Smem* sm, GrayRun& g) {
    *reinterpret_cast<uint2*>(sm->lut + lane * 8) = *reinterpret_cast<const uint2*>(a.p2 + lane * 8);
    gray_load(a, q, max(tb - 1, 0), g);
    g.carryA = g.nextA;
    g.carryB = g.nextB;
    gray_load(a, q, tb + lane, g);
}
__device__ __forceinline__ void p2_block(const Args8& a, const Pair& q, int t0, int lane, P2Smem* sm, GrayRun& g) {
    const int gA = g.nextA, gB = g.nextB;
    gray_load(a, q, t0 + 32 + lane, g);
    int prA = __shfl_up_sync(0xffffffffu, gA, 1), prB = __shfl_up_sync(0xffffffffu, gB, 1);
    if (lane == 0) { prA = g.carryA; prB = g.carryB; }
    g.carryA = __shfl_sync(0xffffffffu, gA, 31);
    g.carryB = __shfl_sync(0xffffffffu, gB, 31);
    __syncwarp();  // the last block's words are read (and, at first, the table is written)
    uint32_t v = (uint32_t)sm->lut[abs(gA - prA)] | ((uint32_t)sm->lut[abs(gB - prB)] << 16);
    // a scanline's first pixel: P2 = 0 (with L' = 0, every delta is 0)
    if (t0 + lane == 0) v = 0;
    sm->w[lane] = v;
    __syncwarp();
}
// P2 of the KG steps from u0 (a multiple of KG) of the block.
template <int KG>
__device__ __forceinline__ void p2_group(const P2Smem* sm, int u0, uint32_t (&p2)[KG]) {
    if constexpr (KG % 4 == 0) {
#pragma unroll
        for (int v = 0; v < KG; v += 4) {
            const uint4 t = *reinterpret_cast<const uint4*>(sm->w + u0 + v);
            p2[v] = t.x; p2[v + 1] = t.y; p2[v + 2] = t.z; p2[v + 3] = t.w;
        }
    } else {
#pragma unroll
        for (int v = 0; v < KG; ++v) p2[v] = sm->w[u0 + v];
    }
}
// Every disparity of the range is valid for every pixel of the steps [t0, t0 + 32) (default ranges:
// d0 <= d < min(dmax, x + 1), x - d < w).
__device__ __forceinline__ bool clean_block(const Args8& a, const Pair& q, int dx, int t0) {
    const int xa = q.xA + t0 * dx, xb = q.xB + t0 * dx, xe = 31 * dx;
    const int lo = min(xa, xb) + min(xe, 0), hi = max(xa, xb) + max(xe, 0);
    return a.def_ranges && lo >= a.dmax - 1 && hi <= a.w - 1 + min(a.d0, 0);
}

template <int DP>
__device__ __forceinline__ void pad_words(const Args8& a, int lane, uint32_t (&pad)[Geo<DP>::W]) {
    constexpr int W = Geo<DP>::W;
#pragma unroll
    for (int k = 0; k < W; ++k) pad[k] = lane * W + k >= a.D ? kPad2 : kBias2;
}

// Copies of whole groups into a ring of groups of KG steps, `narr` arrays of equal shape per step
// (slot layout: [array][A, B][DP]): lane l brings 16 bytes, of step `sub` of its copy instruction.
template <int DP>
struct Copier {
    using G = Geo<DP>;
    int sub, mylen, it;
    int64_t bstep, off;  // byte step of a pixel step; byte offset of the lane's next chunk in every array
    __device__ __forceinline__ void init(const Pair& q, int tb, int lane) {
        sub = lane / (2 * G::CH);
        const int r = lane - sub * (2 * G::CH);
        const bool isB = r >= G::CH;
        mylen = sub < G::SPI ? (isB ? q.lenB : q.lenA) : 0;
        bstep = (int64_t)q.step * DP;
        off = (int64_t)(isB ? q.pB : q.pA) * DP + (tb + sub) * bstep + (isB ? r - G::CH : r) * 16;
        it = tb;
    }
    // dst: the slot of the group's first step plus this lane's place (place()); SLOT: bytes per step
    template <int SLOT, int NARR, int KG, typename BASE>
    __device__ __forceinline__ void group(uint8_t* dst, BASE base) {
        // (a group shorter than a copy instruction's steps leaves its upper lanes idle)
        constexpr int STEP = KG < G::SPI ? KG : G::SPI;
#pragma unroll
        for (int i = 0; i < KG; i += STEP) {
            if (sub < STEP && it + i + sub < mylen) {
#pragma unroll
                for (int b = 0; b < NARR; ++b) cp16(dst + i * SLOT + b * 2 * DP, base(b) + off);
            }
            off += STEP * bstep;
        }
        it += KG;
        cp_commit();
    }
    template <int SLOT>
    __device__ __forceinline__ static int place(int lane) {
        return lane / (2 * G::CH) * SLOT + lane % (2 * G::CH) * 16;
    }
};

template <int DP>
__device__ __forceinline__ void store_deltas(uint8_t* pa, uint8_t* pb, bool doA, bool doB,
                                             const uint32_t (&dl)[Geo<DP>::W]) {
    constexpr int W = Geo<DP>::W;
    uint32_t u[W / 2];
#pragma unroll
    for (int i = 0; i < W / 2; ++i) u[i] = dl[2 * i + 1] * 256u + dl[2 * i];
    if constexpr (W == 2) {
        if (doA) *reinterpret_cast<uint16_t*>(pa) = (uint16_t)u[0];
        if (doB) *reinterpret_cast<uint16_t*>(pb) = (uint16_t)(u[0] >> 16);
    } else if constexpr (W == 4) {
        if (doA) *reinterpret_cast<uint32_t*>(pa) = prmt(u[0], u[1], 0x5410);
        if (doB) *reinterpret_cast<uint32_t*>(pb) = prmt(u[0], u[1], 0x7632);
    } else {
        if (doA) *reinterpret_cast<uint2*>(pa) = make_uint2(prmt(u[0], u[1], 0x5410), prmt(u[2], u[3], 0x5410));
        if (doB) *reinterpret_cast<uint2*>(pb) = make_uint2(prmt(u[0], u[1], 0x7632), prmt(u[2], u[3], 0x7632));
    }
}

// ---- first phase: one warp, scanlines s and s + 1 of direction (dx, dy), deltas to `out`
//
// Steps go in groups of kFirstG: a group's costs are one cp.async group, waited for once and read from
// the ring together, so the steps of a group hold nothing but the recurrence and the stores.
constexpr int kFirstG = 8;
template <int DP>
__host__ __device__ constexpr int first_groups() { return DP >= 192 ? 3 : 4; }  // ring depth in groups
template <int DP>
__host__ __device__ constexpr int first_bytes() { return (int)sizeof(P2Smem) + first_groups<DP>() * kFirstG * 2 * DP + kTail; }

template <int DP>
__device__ __forceinline__ void run_first8(const Args8& a, uint8_t* smem, int dx, int dy, int s, int nscan,
                                           uint8_t* out) {
    using G = Geo<DP>;
    constexpr int W = G::W, SLOT = 2 * DP, NG = first_groups<DP>(), KG = kFirstG;
    P2Smem* sm = reinterpret_cast<P2Smem*>(smem);
    uint8_t* ring = smem + sizeof(P2Smem);
    const int lane = threadIdx.x & 31;
    const Pair q = pair_start(a, dx, dy, s, nscan);
    if (q.maxlen == 0) return;
    Copier<DP> cp;
    cp.init(q, 0, lane);
    uint8_t* dst = ring + Copier<DP>::template place<SLOT>(lane);
    auto base = [&](int) { return a.vol; };
#pragma unroll
    for (int t = 0; t < NG - 1; ++t) cp.template group<SLOT, 1, KG>(dst + t * KG * SLOT, base);
    uint32_t pad[W];
    pad_words<DP>(a, lane, pad);
    Chain<W> st;
    chain_init(st);
    GrayRun g;
    gray_init(a, q, 0, lane, sm, g);
    const uint32_t p1x2 = (uint32_t)a.P1 * 0x00010001u;
    const uint8_t* rd = ring + lane * W;
    // output addresses: pointers per group of steps up to 128 padded disparities, 32-bit offsets (the
    // host checks the volume's size) beyond, whichever measured faster (first phase per frame, pointers
    // / offsets: 640x480 D64 48 / 58 us, 1280x720 D128 148 / 148, eight paths at 1920x1080 D256
    // 1.30 / 1.27 ms)
    constexpr bool PTR = DP <= 128;
    uint8_t* pa = out + (size_t)q.pA * DP + lane * W;
    uint8_t* pb = out + (size_t)q.pB * DP + lane * W;
    const int64_t pstep = (int64_t)q.step * DP;
    uint32_t oa = (uint32_t)q.pA * DP + lane * W, ob = (uint32_t)q.pB * DP + lane * W;
    const uint32_t ostep = (uint32_t)(q.step * DP);
    const bool act = G::AL == 32 || lane < G::AL;
    int slot = 0;
    auto groups = [&](auto clean, auto full, int t0) {
#pragma unroll 1
        for (int u0 = 0; u0 < 32; u0 += KG) {
            const int tb = t0 + u0;
            if (!decltype(full)::value && tb >= q.maxlen) break;
            cp_wait<NG - 2>();
            __syncwarp();
            cp.template group<SLOT, 1, KG>(dst + (slot == 0 ? NG - 1 : slot - 1) * (KG * SLOT), base);
            const uint8_t* sl = rd + slot * (KG * SLOT);
            Raw<DP> raw[KG];
            uint32_t p2[KG];
            p2_group<KG>(sm, u0, p2);
#pragma unroll
            for (int v = 0; v < KG; ++v) {
                raw[v] = load_raw<DP>(sl + v * SLOT);
            }
#pragma unroll
            for (int v = 0; v < KG; ++v) {
                uint32_t c[W], dl[W];
                path_step<DP, decltype(clean)::value>(st, raw[v], pad, p1x2, p2[v], lane, c, dl);
                const bool doA = act && (decltype(full)::value || tb + v < q.lenA);
                const bool doB = act && (decltype(full)::value || tb + v < q.lenB);
                if constexpr (PTR) {
                    store_deltas<DP>(pa + v * pstep, pb + v * pstep, doA, doB, dl);
                } else {
                    store_deltas<DP>(out + oa, out + ob, doA, doB, dl);
                    oa += ostep;
                    ob += ostep;
                }
            }
            if constexpr (PTR) {
                pa += KG * pstep;
                pb += KG * pstep;
            }
            slot = slot == NG - 1 ? 0 : slot + 1;
        }
    };
    for (int t0 = 0; t0 < q.maxlen; t0 += 32) {
        p2_block(a, q, t0, lane, sm, g);
        if (t0 + 32 > q.minlen) groups(std::false_type(), std::false_type(), t0);
        else if (clean_block(a, q, dx, t0)) groups(std::true_type(), std::true_type(), t0);
        else groups(std::false_type(), std::true_type(), t0);
    }
    cp_wait<0>();
    __syncwarp();
}

// ---- last sweep: the sums n * C + deltas of NIN first-phase directions and of this sweep, the WTA
//
// PS: two deltas of one voxel fit a byte, so two arrays are added before they are widened.
template <int NIN>
__host__ __device__ constexpr uint32_t sum_bias() { return kBias * (NIN + 1); }
template <int NIN>
__host__ __device__ constexpr uint32_t sum_inf() { return (kBias + kInvalid) * (NIN + 1); }

// The deltas of NIN arrays at sl (layout [array][A, B][DP]); with PS in pairs, added as bytes.
template <int DP, int NIN, bool PS>
struct Deltas {
    static constexpr int N = PS ? (NIN + 1) / 2 : NIN;
    Raw<DP> r[N];
};
template <int DP, int NIN, bool PS>
__device__ __forceinline__ Deltas<DP, NIN, PS> load_deltas(const uint8_t* sl) {
    Deltas<DP, NIN, PS> d;
#pragma unroll
    for (int b = 0; b < NIN; ++b) {
        const Raw<DP> r = load_raw<DP>(sl + b * 2 * DP);
        if (PS && (b & 1)) {
#pragma unroll
            for (int i = 0; i < Raw<DP>::N; ++i) {
                d.r[b / 2].a[i] += r.a[i];
                d.r[b / 2].b[i] += r.b[i];
            }
        } else {
            d.r[PS ? b / 2 : b] = r;
        }
    }
    return d;
}
template <int DP, int NIN, bool PS>
__device__ __forceinline__ void add_deltas(const Deltas<DP, NIN, PS>& d, uint32_t (&sum)[Geo<DP>::W]) {
    constexpr int W = Geo<DP>::W;
#pragma unroll
    for (int b = 0; b < Deltas<DP, NIN, PS>::N; ++b) {
        uint32_t e[W / 2];
        interleave<DP>(d.r[b], e);
#pragma unroll
        for (int i = 0; i < W / 2; ++i) {
            sum[2 * i] += e[i] & 0x00FF00FFu;
            sum[2 * i + 1] += prmt(e[i], 0u, 0x4341);
        }
    }
}

// The sums of one step into the WTA buffer: rows v (A) and 16 + v (B), two consecutive disparities a word.
template <int DP, int NIN>
__device__ __forceinline__ void put_sums(const Args8& a, const Pair& q, uint32_t* s_wta, int v, int t, int lane, bool act,
                                         const uint32_t (&sum)[Geo<DP>::W]) {
    using G = Geo<DP>;
    constexpr int W = G::W;
    if (!act) return;
    uint32_t* wa = s_wta + v * G::RS + lane * (W / 2);
    uint32_t* wb = wa + 16 * G::RS;
    uint32_t oa[W / 2], ob[W / 2];
#pragma unroll
    for (int i = 0; i < W / 2; ++i) {
        oa[i] = prmt(sum[2 * i], sum[2 * i + 1], 0x5410);
        ob[i] = prmt(sum[2 * i], sum[2 * i + 1], 0x7632);
    }
    if constexpr (W == 2) {
        wa[0] = oa[0];
        wb[0] = ob[0];
    } else if constexpr (W == 4) {
        *reinterpret_cast<uint2*>(wa) = make_uint2(oa[0], oa[1]);
        *reinterpret_cast<uint2*>(wb) = make_uint2(ob[0], ob[1]);
    } else {
        *reinterpret_cast<uint4*>(wa) = make_uint4(oa[0], oa[1], oa[2], oa[3]);
        *reinterpret_cast<uint4*>(wb) = make_uint4(ob[0], ob[1], ob[2], ob[3]);
    }
    if (a.sum) {
        constexpr uint32_t inf = sum_inf<NIN>() * 0x00010001u, bias = sum_bias<NIN>() * 0x00010001u;
#pragma unroll
        for (int i = 0; i < W / 2; ++i) {
            const size_t o = (size_t)lane * (W / 2) + i;
            if (t < q.lenA)
                a.sum[(size_t)(q.pA + t * q.step) * (DP / 2) + o] = (oa[i] - bias) | __vcmpgeu2(oa[i], inf);
            if (t < q.lenB)
                a.sum[(size_t)(q.pB + t * q.step) * (DP / 2) + o] = (ob[i] - bias) | __vcmpgeu2(ob[i], inf);
        }
    }
}

// The WTA of the block of 16 steps at tb: lane l takes step tb + l % 16 of scanline A (l < 16) or B (none
// where B repeats A, an odd last scanline: the sub-pixel telemetry counts a pixel once).
template <int DP, int NIN>
__device__ __forceinline__ void wta_block(const Args8& a, const Pair& q, uint32_t* s_wta, int tb, int lane) {
    const int t = tb + (lane & 15);
    const bool b = lane >= 16;
    if (t < (b ? q.lenB : q.lenA) && !(b && q.pB == q.pA))
        wta_row<DP / 2, sum_inf<NIN>(), sum_bias<NIN>()>(a.wta, a.d0, a.D, s_wta + lane * Geo<DP>::RS,
                                                         (b ? q.pB : q.pA) + t * q.step);
}

// Bands of steps [t_begin, t_end): the chains' path values enter and leave through a.carry.
__device__ __forceinline__ bool band_limits(const Args8& a, Pair& q, int& tb0) {
    tb0 = a.t_begin;
    const bool carry_out = a.t_end < q.maxlen;
    q.lenA = min(q.lenA, a.t_end);
    q.lenB = min(q.lenB, a.t_end);
    q.maxlen = min(q.maxlen, a.t_end);
    q.minlen = min(q.minlen, a.t_end);
    return carry_out;
}
template <int DP>
__device__ __forceinline__ void band_load(const Args8& a, int s, int lane, uint32_t p1x2, Chain<Geo<DP>::W>& st) {
    const uint32_t* cs = a.carry + (size_t)(s >> 1) * Geo<DP>::W * 32 + lane;
#pragma unroll
    for (int k = 0; k < Geo<DP>::W; ++k) {
        st.L[k] = __ldcg(cs + k * 32);
        st.q[k] = st.L[k] + p1x2;
    }
    chain_reduce(st);
}
template <int DP>
__device__ __forceinline__ void band_store(const Args8& a, int s, int lane, const Chain<Geo<DP>::W>& st) {
    uint32_t* cs = a.carry + (size_t)(s >> 1) * Geo<DP>::W * 32 + lane;
#pragma unroll
    for (int k = 0; k < Geo<DP>::W; ++k) __stcg(cs + k * 32, st.L[k]);
}

// One warp per pair of scanlines: rings of NG groups of KG steps.
template <int DP, int NIN, int KG, int NG>
__host__ __device__ constexpr int last_bytes() {
    return (int)sizeof(P2Smem) + Geo<DP>::wta_words * 4 + NG * KG * (1 + NIN) * 2 * DP + kTail;
}
template <int DP, int NIN, int KG, int NG, bool PS, bool BAND>
__device__ __forceinline__ void run_last8(const Args8& a, const uint8_t* const* in, uint8_t* smem, int dx, int dy, int s,
                                          int nscan) {
    using G = Geo<DP>;
    constexpr int W = G::W, NARR = 1 + NIN, SLOT = NARR * 2 * DP;
    static_assert(16 % KG == 0, "a WTA block is whole groups");
    P2Smem* sm = reinterpret_cast<P2Smem*>(smem);
    uint32_t* s_wta = reinterpret_cast<uint32_t*>(smem + sizeof(P2Smem));
    uint8_t* ring = smem + sizeof(P2Smem) + G::wta_words * 4;
    const int lane = threadIdx.x & 31;
    Pair q = pair_start(a, dx, dy, s, nscan);
    int tb0 = 0;
    bool carry_out = false;
    if constexpr (BAND) carry_out = band_limits(a, q, tb0);
    if (q.maxlen <= tb0) return;
    Copier<DP> cp;
    cp.init(q, tb0, lane);
    uint8_t* dst = ring + Copier<DP>::template place<SLOT>(lane);
    auto base = [&](int b) { return b == 0 ? a.vol : in[b - 1]; };
#pragma unroll
    for (int t = 0; t < NG - 1; ++t) cp.template group<SLOT, NARR, KG>(dst + t * KG * SLOT, base);
    uint32_t pad[W];
    pad_words<DP>(a, lane, pad);
    const uint32_t p1x2 = (uint32_t)a.P1 * 0x00010001u;
    Chain<W> st;
    chain_init(st);
    if constexpr (BAND)
        if (tb0 > 0) band_load<DP>(a, s, lane, p1x2, st);
    GrayRun g;
    gray_init(a, q, tb0, lane, sm, g);
    const uint8_t* rd = ring + lane * W;
    const bool act = G::AL == 32 || lane < G::AL;
    int slot = 0;
    auto groups = [&](auto clean, int t0) {
#pragma unroll 1
        for (int u0 = 0; u0 < 32; u0 += KG) {
            const int tb = t0 + u0;
            if (tb >= q.maxlen) break;
            cp_wait<NG - 2>();
            __syncwarp();
            cp.template group<SLOT, NARR, KG>(dst + (slot == 0 ? NG - 1 : slot - 1) * (KG * SLOT), base);
            const uint8_t* sl = rd + slot * (KG * SLOT);
            // everything the group reads from the ring first: the sums' stores below may not be
            // reordered with later loads
            Raw<DP> raw[KG];
            Deltas<DP, NIN, PS> de[KG];
            uint32_t p2[KG];
            p2_group<KG>(sm, u0, p2);
#pragma unroll
            for (int v = 0; v < KG; ++v) {
                raw[v] = load_raw<DP>(sl + v * SLOT);
                de[v] = load_deltas<DP, NIN, PS>(sl + v * SLOT + 2 * DP);
            }
#pragma unroll
            for (int v = 0; v < KG; ++v) {
                uint32_t c[W], dl[W], sum[W];
                path_step<DP, decltype(clean)::value>(st, raw[v], pad, p1x2, p2[v], lane, c, dl);
#pragma unroll
                for (int k = 0; k < W; ++k) sum[k] = c[k] * (uint32_t)(NIN + 1) + dl[k];
                add_deltas<DP, NIN, PS>(de[v], sum);
                put_sums<DP, NIN>(a, q, s_wta, (u0 + v) & 15, tb + v, lane, act, sum);
            }
            slot = slot == NG - 1 ? 0 : slot + 1;
            if (((u0 + KG) & 15) == 0 || tb + KG >= q.maxlen) {
                __syncwarp();
                wta_block<DP, NIN>(a, q, s_wta, t0 + (u0 & 16), lane);
                __syncwarp();
            }
        }
    };
    for (int t0 = tb0; t0 < q.maxlen; t0 += 32) {
        p2_block(a, q, t0, lane, sm, g);
        if (clean_block(a, q, dx, t0)) groups(std::true_type(), t0);
        else groups(std::false_type(), t0);
    }
    if constexpr (BAND)
        if (carry_out) band_store<DP>(a, s, lane, st);
    cp_wait<0>();
    __syncwarp();
}

// Two warps per pair of scanlines: warp 0 runs the recurrence and hands each step's n * C + delta to
// warp 1, which adds the other directions' deltas and runs the WTA.  Steps change hands in segments of
// KG steps through two shared buffers: warp 0 arrives on FULL[slot] once a segment is written and waits on
// FREE[slot] before it writes the slot again, warp 1 the other way round.  Both walk the same number of
// segments (one pair per block), so every barrier generation is completed by one arrival of each warp.
// Barrier ids are immediates (a register id would make the compiler reserve all sixteen) and the kernel
// has no other block barrier.
template <int DP, int NIN, int KG, int NGP, int NGC>
struct Split8 {
    static constexpr int ring_p = NGP * KG * 2 * DP + kTail;
    static constexpr int ring_c = NGC * KG * NIN * 2 * DP + kTail;
    static constexpr int part = 2 * KG * DP * 4;
    static constexpr int bytes = (int)sizeof(P2Smem) + Geo<DP>::wta_words * 4 + part + ring_p + ring_c;
};
template <int ID>
__device__ __forceinline__ void nbar_sync() { asm volatile("bar.sync %0, 64;\n" ::"n"(ID) : "memory"); }
template <int ID>
__device__ __forceinline__ void nbar_arrive() { asm volatile("bar.arrive %0, 64;\n" ::"n"(ID) : "memory"); }
// barrier BASE + slot for a slot of two
template <int BASE, bool SYNC>
__device__ __forceinline__ void nbar(int slot) {
    if (slot) {
        if (SYNC) nbar_sync<BASE + 1>();
        else nbar_arrive<BASE + 1>();
    } else {
        if (SYNC) nbar_sync<BASE>();
        else nbar_arrive<BASE>();
    }
}
constexpr int kSeg = 2;
constexpr int kFull = 0, kFree = kSeg;

template <int DP, int NIN, int KG, int NGP, int NGC, bool PS, bool BAND>
__global__ void __launch_bounds__(64) sgm8_last_split_kernel(Args8 a, In8 in, int dx, int dy, int nscan) {
    using G = Geo<DP>;
    using S = Split8<DP, NIN, KG, NGP, NGC>;
    constexpr int W = G::W;
    static_assert(16 % KG == 0, "a WTA block is whole segments");
    extern __shared__ __align__(16) uint8_t s8[];
    P2Smem* sm = reinterpret_cast<P2Smem*>(s8);
    uint32_t* s_wta = reinterpret_cast<uint32_t*>(s8 + sizeof(P2Smem));
    uint32_t* s_part = s_wta + G::wta_words;
    uint8_t* ring_p = s8 + sizeof(P2Smem) + G::wta_words * 4 + S::part;
    uint8_t* ring_c = ring_p + S::ring_p;
    const int lane = threadIdx.x & 31;
    const int s = 2 * (int)blockIdx.x;
    Pair q = pair_start(a, dx, dy, s, nscan);
    int tb0 = 0;
    bool carry_out = false;
    if constexpr (BAND) carry_out = band_limits(a, q, tb0);
    if (q.maxlen <= tb0) return;  // the whole block (one pair)
    const int nseg = (q.maxlen - tb0 + KG - 1) / KG;
    const bool act = G::AL == 32 || lane < G::AL;
    uint32_t* part = s_part + lane * W;
    Copier<DP> cp;
    cp.init(q, tb0, lane);
    if (threadIdx.x < 32) {
        constexpr int SLOT = 2 * DP;
        uint8_t* dst = ring_p + Copier<DP>::template place<SLOT>(lane);
        auto base = [&](int) { return a.vol; };
#pragma unroll
        for (int t = 0; t < NGP - 1; ++t) cp.template group<SLOT, 1, KG>(dst + t * KG * SLOT, base);
        uint32_t pad[W];
        pad_words<DP>(a, lane, pad);
        const uint32_t p1x2 = (uint32_t)a.P1 * 0x00010001u;
        Chain<W> st;
        chain_init(st);
        if constexpr (BAND)
            if (tb0 > 0) band_load<DP>(a, s, lane, p1x2, st);
        GrayRun g;
        gray_init(a, q, tb0, lane, sm, g);
        const uint8_t* rd = ring_p + lane * W;
        int slot = 0;
        auto groups = [&](auto clean, int t0) {
#pragma unroll 1
            for (int u0 = 0; u0 < 32; u0 += KG) {
                const int tb = t0 + u0;
                if (tb >= q.maxlen) break;
                cp_wait<NGP - 2>();
                __syncwarp();
                cp.template group<SLOT, 1, KG>(dst + (slot == 0 ? NGP - 1 : slot - 1) * (KG * SLOT), base);
                const uint8_t* sl = rd + slot * (KG * SLOT);
                Raw<DP> raw[KG];
                uint32_t p2[KG];
                p2_group<KG>(sm, u0, p2);
#pragma unroll
                for (int v = 0; v < KG; ++v) {
                    raw[v] = load_raw<DP>(sl + v * SLOT);
                }
                const int seg = (tb - tb0) / KG, sb = seg % kSeg;
                if (seg >= kSeg) nbar<kFree, true>(sb);
#pragma unroll
                for (int v = 0; v < KG; ++v) {
                    uint32_t c[W], dl[W];
                    path_step<DP, decltype(clean)::value>(st, raw[v], pad, p1x2, p2[v], lane, c, dl);
                    if (act) {
                        uint32_t* o = part + (sb * KG + v) * DP;
#pragma unroll
                        for (int k = 0; k < W; ++k) c[k] = c[k] * (uint32_t)(NIN + 1) + dl[k];
                        if constexpr (W == 2) *reinterpret_cast<uint2*>(o) = make_uint2(c[0], c[1]);
                        else {
#pragma unroll
                            for (int k = 0; k < W; k += 4)
                                *reinterpret_cast<uint4*>(o + k) = make_uint4(c[k], c[k + 1], c[k + 2], c[k + 3]);
                        }
                    }
                }
                __threadfence_block();
                nbar<kFull, false>(sb);
                slot = slot == NGP - 1 ? 0 : slot + 1;
            }
        };
        for (int t0 = tb0; t0 < q.maxlen; t0 += 32) {
            p2_block(a, q, t0, lane, sm, g);
            if (clean_block(a, q, dx, t0)) groups(std::true_type(), t0);
            else groups(std::false_type(), t0);
        }
        if constexpr (BAND)
            if (carry_out) band_store<DP>(a, s, lane, st);
    } else {
        constexpr int SLOT = NIN * 2 * DP;
        uint8_t* dst = ring_c + Copier<DP>::template place<SLOT>(lane);
        auto base = [&](int b) { return in.d[b]; };
#pragma unroll
        for (int t = 0; t < NGC - 1; ++t) cp.template group<SLOT, NIN, KG>(dst + t * KG * SLOT, base);
        const uint8_t* rd = ring_c + lane * W;
        int slot = 0;
#pragma unroll 1
        for (int seg = 0; seg < nseg; ++seg) {
            const int tb = tb0 + seg * KG, sb = seg % kSeg;
            cp_wait<NGC - 2>();
            __syncwarp();
            cp.template group<SLOT, NIN, KG>(dst + (slot == 0 ? NGC - 1 : slot - 1) * (KG * SLOT), base);
            const uint8_t* sl = rd + slot * (KG * SLOT);
            // the segment's reads come first, half a segment at a time: the sums' stores may not be
            // reordered with later loads
            constexpr int H = KG >= 4 ? 4 : KG;
            Deltas<DP, NIN, PS> de[H];
#pragma unroll
            for (int v = 0; v < H; ++v) de[v] = load_deltas<DP, NIN, PS>(sl + v * SLOT);
            nbar<kFull, true>(sb);
#pragma unroll
            for (int h = 0; h < KG; h += H) {
                uint32_t sum[H][W];
#pragma unroll
                for (int v = 0; v < H; ++v) {
                    const uint32_t* o = part + (sb * KG + h + v) * DP;
                    if constexpr (W == 2) {
                        const uint2 x = *reinterpret_cast<const uint2*>(o);
                        sum[v][0] = x.x; sum[v][1] = x.y;
                    } else {
#pragma unroll
                        for (int k = 0; k < W; k += 4) {
                            const uint4 x = *reinterpret_cast<const uint4*>(o + k);
                            sum[v][k] = x.x; sum[v][k + 1] = x.y; sum[v][k + 2] = x.z; sum[v][k + 3] = x.w;
                        }
                    }
                    if (h > 0) de[v] = load_deltas<DP, NIN, PS>(sl + (h + v) * SLOT);
                }
#pragma unroll
                for (int v = 0; v < H; ++v) {
                    add_deltas<DP, NIN, PS>(de[v], sum[v]);
                    put_sums<DP, NIN>(a, q, s_wta, (tb + h + v) & 15, tb + h + v, lane, act, sum[v]);
                }
            }
            __threadfence_block();
            if (seg + kSeg < nseg) nbar<kFree, false>(sb);
            slot = slot == NGC - 1 ? 0 : slot + 1;
            if (((tb + KG) & 15) == 0 || seg == nseg - 1) {
                __syncwarp();
                wta_block<DP, NIN>(a, q, s_wta, tb & ~15, lane);
                __syncwarp();
            }
        }
    }
    cp_wait<0>();
}

// One warp per block: chains of different lengths end independently.
template <int DP>
__global__ void __launch_bounds__(32) sgm8_first_kernel(Args8 a, Dirs8 tab) {
    extern __shared__ __align__(16) uint8_t s8[];
    int d = 0;
#pragma unroll
    for (int i = 1; i < kMaxIn; ++i)
        if (i < tab.n && (int)blockIdx.x >= tab.warp_begin[i]) d = i;
    const int s = 2 * ((int)blockIdx.x - tab.warp_begin[d]);
    run_first8<DP>(a, s8, tab.dx[d], tab.dy[d], s, tab.nscan[d], tab.out[d]);
}

template <int DP, int NIN, int KG, int NG, bool PS, bool BAND>
__global__ void __launch_bounds__(32) sgm8_last_kernel(Args8 a, In8 in, int dx, int dy, int nscan) {
    extern __shared__ __align__(16) uint8_t s8[];
    run_last8<DP, NIN, KG, NG, PS, BAND>(a, in.d, s8, dx, dy, 2 * (int)blockIdx.x, nscan);
}

int nscan8(int w, int h, int dx, int dy) { return dy == 0 ? h : (dx == 0 ? w : w + h - 1); }

// adaptive_p2 (common.cuh) on the host, the same single-precision steps.
int host_p2(const SgmPen& p, int dI) {
    int P2 = p.P2_base;
    if (p.adaptive) {
        if (p.piecewise) {
            if (dI >= p.t2) P2 = p.P2_base / 4;
            else if (dI >= p.t1) P2 = p.P2_base / 2;
        } else {
            const volatile float scaled = p.alpha * (float)dI;
            const volatile float den = 1.f + scaled;
            const volatile float quot = (float)p.P2_base / den;
            const volatile float up = quot + 0.5f;
            P2 = (int)up;
        }
    }
    return std::max(P2, p.P1 + 1);
}

Args8 make_args8(const SgmLaunch& l) {
    Args8 a{};
    a.w = l.w; a.h = l.h; a.d0 = l.d0; a.D = l.D; a.dmax = l.d0 + l.D;
    a.def_ranges = l.default_ranges;
    a.P1 = l.pen.P1;
    for (int i = 0; i < 256; ++i) a.p2[i] = (uint8_t)host_p2(l.pen, i);
    a.gray = l.gray;
    a.vol = reinterpret_cast<const uint8_t*>(l.cvol);
    a.wta = WtaOut{l.disp, l.best, l.second, l.subpixel, l.sp_method, l.sp_param, l.sp_tel};
    a.sum = l.sum;
    a.t_begin = 0;
    a.t_end = 0x7FFFFFFF;
    return a;
}

int max_p2(const SgmPen& p) { return p.P2_base > p.P1 + 1 ? p.P2_base : p.P1 + 1; }

template <typename F>
cudaError_t by_dp(int Dp, F f) {
    switch (Dp) {
        case 64: return f(std::integral_constant<int, 64>());
        case 128: return f(std::integral_constant<int, 128>());
        case 192: return f(std::integral_constant<int, 192>());
        case 256: return f(std::integral_constant<int, 256>());
        default: return cudaErrorInvalidValue;
    }
}

// The device's SMs, the shared memory of one and what each block reserves of it (bytes).
struct SmShare {
    int count;
    size_t smem, reserved;
};
SmShare sm_share() {
    int dev = 0, nsm = 0, per_sm = 0, reserved = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev) != cudaSuccess) {
        cudaGetLastError();
        return SmShare{148, 228 * 1024, 1024};
    }
    return SmShare{nsm, (size_t)per_sm, (size_t)reserved};
}

// Blocks of `bytes` shared memory the device holds at once.
int blocks_at_once(size_t bytes) {
    const SmShare sm = sm_share();
    return sm.count * (int)(sm.smem / (bytes + sm.reserved));
}

template <int DP, int NIN, bool PS, bool BAND>
cudaError_t launch_last_t(const Args8& a, const In8& in, int dx, int dy, int nscan, cudaStream_t st) {
    const int blocks = (nscan + 1) / 2;
    // two warps per pair where every pair is resident at once in that form, else one
    constexpr int SG = NIN == 3 && DP <= 128 ? 8 : 4, NGP = DP == 256 ? 2 : 3, NGC = DP == 192 && NIN == 3 ? 3 : 2;
    using S = Split8<DP, NIN, SG, NGP, NGC>;
    if (blocks <= blocks_at_once(S::bytes)) {
        auto kern = sgm8_last_split_kernel<DP, NIN, SG, NGP, NGC, PS, BAND>;
        const size_t smem = S::bytes;
        const cudaError_t e = allow_dynamic_smem(kern, smem);
        if (e != cudaSuccess) return e;
        kern<<<blocks, 64, smem, st>>>(a, in, dx, dy, nscan);
        return cudaGetLastError();
    }
    // steps per group: four keep a group's loads long, two where four leave too few blocks on an SM (Fast
    // 1920x1080, four / two, us: D128 260 / 295, D192 519 / 449; D256 two / one 438 / 512)
    constexpr int KG = DP == 256 ? (NIN == 3 ? 2 : 1) : DP == 192 ? 2 : (NIN == 3 ? 4 : 2), NG = 3;
    auto kern = sgm8_last_kernel<DP, NIN, KG, NG, PS, BAND>;
    const size_t smem = last_bytes<DP, NIN, KG, NG>();
    const cudaError_t e = allow_dynamic_smem(kern, smem);
    if (e != cudaSuccess) return e;
    kern<<<blocks, 32, smem, st>>>(a, in, dx, dy, nscan);
    return cudaGetLastError();
}

template <bool BAND>
cudaError_t launch_last_any(const SgmLaunch& l, const Args8& a, int dx, int dy, int nin, const uint8_t* const* in,
                            cudaStream_t st) {
    if (nin != 3 && (nin != 7 || BAND)) return cudaErrorInvalidValue;
    In8 t{};
    for (int i = 0; i < nin; ++i) t.d[i] = in[i];
    const int nscan = nscan8(l.w, l.h, dx, dy);
    const bool ps = 2 * max_p2(l.pen) <= 255;
    return by_dp(l.Dp, [&](auto dp) -> cudaError_t {
        constexpr int DP = decltype(dp)::value;
        if (nin == 3)
            return ps ? launch_last_t<DP, 3, true, BAND>(a, t, dx, dy, nscan, st)
                      : launch_last_t<DP, 3, false, BAND>(a, t, dx, dy, nscan, st);
        if constexpr (!BAND)
            return ps ? launch_last_t<DP, 7, true, false>(a, t, dx, dy, nscan, st)
                      : launch_last_t<DP, 7, false, false>(a, t, dx, dy, nscan, st);
        return cudaErrorInvalidValue;
    });
}

}  // namespace

bool sgm8_supported(int Dp, const SgmPen& pen) { return Dp <= 256 && Dp % 64 == 0 && max_p2(pen) <= (int)kMaxP2; }

size_t sgm8_carry_words(int w, int Dp) { return (size_t)((w + 1) / 2) * 32 * ((Dp >= 192 ? 8 : Dp / 32)); }

cudaError_t launch_sgm8_first(const SgmLaunch& l, int ndir, const int (*dirs)[2], uint8_t* const* out,
                              cudaStream_t st) {
    if (ndir < 1 || ndir > kMaxIn || !sgm8_supported(l.Dp, l.pen)) return cudaErrorInvalidValue;
    const Args8 a = make_args8(l);
    Dirs8 tab{};
    tab.n = ndir;
    for (int i = 0; i < ndir; ++i) {
        tab.dx[i] = dirs[i][0];
        tab.dy[i] = dirs[i][1];
        tab.out[i] = out[i];
        tab.nscan[i] = nscan8(l.w, l.h, dirs[i][0], dirs[i][1]);
        tab.warp_begin[i + 1] = tab.warp_begin[i] + (tab.nscan[i] + 1) / 2;
    }
    return by_dp(l.Dp, [&](auto dp) -> cudaError_t {
        constexpr int DP = decltype(dp)::value;
        // Frames of many more chains than an SM's four schedulers can step at full rate: eight blocks at a time
        // on each SM, the rest in their turn as chains end, so that fewer rows are open in DRAM and the last
        // chains share an SM with fewer others.  Eight a SM against all that fit, us: 1920x1080 D128 285 / 313,
        // D256 538 / 612, HighQuality D256 1237 / 1282, 2560x1440 D256 1003 / 1028; with fewer chains it loses
        // (1280x720 D128 155 / 147, 1280x1024 D256 381 / 371), as with eight paths below 256 (1280x720 D128
        // 367 / 362).
        const int blocks = tab.warp_begin[ndir];
        size_t smem = first_bytes<DP>();
        const SmShare sm = sm_share();
        if (blocks >= 12 * sm.count && (ndir <= 3 || DP == 256)) smem = std::max(smem, (sm.smem / 8 - sm.reserved) & ~size_t(15));
        const cudaError_t e = allow_dynamic_smem(sgm8_first_kernel<DP>, smem);
        if (e != cudaSuccess) return e;
        sgm8_first_kernel<DP><<<blocks, 32, smem, st>>>(a, tab);
        return cudaGetLastError();
    });
}

cudaError_t launch_sgm8_last(const SgmLaunch& l, int dx, int dy, int nin, const uint8_t* const* in, cudaStream_t st) {
    if (!sgm8_supported(l.Dp, l.pen)) return cudaErrorInvalidValue;
    return launch_last_any<false>(l, make_args8(l), dx, dy, nin, in, st);
}

cudaError_t launch_sgm8_last_band(const SgmLaunch& l, int dx, int dy, int nin, const uint8_t* const* in, int t_begin,
                                  int t_end, uint32_t* carry, cudaStream_t st) {
    if (!sgm8_supported(l.Dp, l.pen) || t_begin < 0 || (t_begin & 31) || t_end <= t_begin || !carry)
        return cudaErrorInvalidValue;
    Args8 a = make_args8(l);
    a.t_begin = t_begin;
    a.t_end = t_end;
    a.carry = carry;
    return launch_last_any<true>(l, a, dx, dy, nin, in, st);
}

}  // namespace apgcu
