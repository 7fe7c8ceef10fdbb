// HighQuality selective refinement, detail::refine_scalar (src/refiner.cpp:42-100).
//
// The reference walks the image in raster order (forward on even passes, backward on odd) and
// updates unreliable pixels in place, so a pixel sees the already-updated values of its causal
// neighbours (left and up forward, right and down backward).
//
// Schedule: a pass is one launch of refine_band_kernel.  A warp owns a band of 32 consecutive
// (pass-order) rows, lane i row i, and walks the columns with lane i one column behind lane i-1:
// at step t lane i updates column t - i, so its up neighbour is what lane i-1 produced at step
// t-1 (one shuffle) and its left neighbour is its own previous value.  The first row of a band
// takes the row above from the band above, eight columns at a time: through the shared memory of the
// thread-block cluster the two bands run in, or between clusters through global memory and a progress
// counter.  The bands run as a wavefront about 48 steps apart and a pass takes about w + 1.5 h steps.
// Every wait is bounded: on timeout the band sets an error flag (read by the host) and stops.  This is
// exactly the reference's read-after-write order.
//
// A band keeps the row above whole in shared memory (5 bytes a column), so frames whose bands do not all
// fit on the device at once that way take a pass in several runs of columns, one launch after another: every
// row of a run comes before the next run's first column, whose left neighbours are then read from the map.
// Frames of more bands than the device holds whatever the columns (740, 23,680 rows) take a pass in groups of
// bands, one launch after another: the band above a group's first has ended, its last row lies in the map.
//
// Measured (one B200, all three passes of HighQuality with their per-pixel kernels): 1920x1080 D256
// 1.97 ms, 1280x720 D128 1.27 ms, where steps with divergent branches, per-step hand-overs by polling
// and per-lane copies took 5.61 and 3.70 ms; a step costs about 300 cycles.
//
// Random draws: a pixel consumes a draw when it is unreliable, has a non-empty range and holds a
// non-negative value at the start of the pass, so its draw index is an exclusive prefix count of
// such pixels in the pass's raster order.  The reference takes draws from one std::mt19937(12345)
// stream through a fresh std::uniform_int_distribution<int>(-r, r) per pass.  A draw maps one
// accepted engine output to a value and skips rejected outputs, each a function of that single
// output, so per radius the value of every output of the (fixed) stream and the rare rejected
// indices are tabulated once, on the host, by the standard library itself: pass `it` then takes
// the q-th accepted output at or after its start position P_it, and P_{it+1} follows on the device
// from the pass's count.  No host work or synchronisation remains per frame.
#include <algorithm>
#include <map>
#include <mutex>
#include <random>
#include <vector>

#include "engine.h"

namespace apgcu {

namespace {

constexpr int kBand = 32;
constexpr int kChunk = 8;        // steps between exchanges (records, row above, progress)
constexpr int kMaxRejected = 64;  // rejected outputs tabulated per radius (expected: none)

__global__ void refine_flags_kernel(int w, int h, const uint8_t* __restrict__ reliable, const int16_t* __restrict__ rmin,
                                    const int16_t* __restrict__ rmax, const float* __restrict__ work, int fwd,
                                    int* __restrict__ flags) {
    const int n = w * h;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i <= n; i += gridDim.x * blockDim.x) {
        if (i == n) { flags[n] = 0; continue; }
        const int f = (!reliable[i] && rmax[i] > rmin[i] && work[i] >= 0.f) ? 1 : 0;
        flags[fwd ? i : n - 1 - i] = f;
    }
}

// Exclusive prefix sum of the flags in place (the draw index of every pixel, and the pass's count
// at index n): three launches without atomics or waits, so the result does not depend on
// scheduling.  A tile is kScanThreads x kScanPer consecutive entries.
constexpr int kScanThreads = 1024, kScanPer = 4, kScanTile = kScanThreads * kScanPer;

// Exclusive prefix of v over the block and the block's total (s_warp: 32 ints).
__device__ __forceinline__ int block_exclusive(int v, int* s_warp, int* total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[wid] = x;
    __syncthreads();
    if (wid == 0) {
        int t = lane < (int)(blockDim.x >> 5) ? s_warp[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        s_warp[lane] = t;
    }
    __syncthreads();
    *total = s_warp[31];
    const int before = wid ? s_warp[wid - 1] : 0;
    __syncthreads();  // s_warp may be reused by the caller
    return before + x - v;
}

__global__ void __launch_bounds__(kScanThreads) scan_tile_sums_kernel(const int* __restrict__ in, int n,
                                                                      int* __restrict__ sums) {
    __shared__ int s_warp[32];
    const size_t base = (size_t)blockIdx.x * kScanTile + (size_t)threadIdx.x * kScanPer;
    int v = 0;
#pragma unroll
    for (int k = 0; k < kScanPer; ++k)
        if (base + k < (size_t)n) v += in[base + k];
    int total = 0;
    block_exclusive(v, s_warp, &total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// One block: the tile sums [0, nt) into exclusive tile offsets, in place.
__global__ void __launch_bounds__(kScanThreads) scan_tile_offsets_kernel(int* sums, int nt) {
    __shared__ int s_warp[32];
    int carry = 0;
    for (int b = 0; b < nt; b += kScanThreads) {
        const int i = b + (int)threadIdx.x;
        const int v = i < nt ? sums[i] : 0;
        int total = 0;
        const int ex = block_exclusive(v, s_warp, &total);
        if (i < nt) sums[i] = carry + ex;
        carry += total;
    }
}

__global__ void __launch_bounds__(kScanThreads) scan_apply_kernel(int* data, int n, const int* __restrict__ offs) {
    __shared__ int s_warp[32];
    const size_t base = (size_t)blockIdx.x * kScanTile + (size_t)threadIdx.x * kScanPer;
    int v[kScanPer];
    int sum = 0;
#pragma unroll
    for (int k = 0; k < kScanPer; ++k) {
        v[k] = base + k < (size_t)n ? data[base + k] : 0;
        sum += v[k];
    }
    int total = 0;
    int run = offs[blockIdx.x] + block_exclusive(sum, s_warp, &total);
#pragma unroll
    for (int k = 0; k < kScanPer; ++k) {
        if (base + k < (size_t)n) data[base + k] = run;
        run += v[k];
    }
}

// Raw index of the q-th accepted output at or after P (rejected indices sorted ascending).
__device__ __forceinline__ unsigned accepted_index(unsigned P, unsigned q, const unsigned* rej, int nrej) {
    unsigned idx = P + q;
    for (int k = 0; k < nrej; ++k) {
        const unsigned r = rej[k];
        if (r < P) continue;
        if (r <= idx) ++idx;
        else break;
    }
    return idx;
}

// Start of pass `it + 1`: the stream position after pass `it`'s count of draws from P[it]; also
// clears the bands' progress counters for the next pass.
__global__ void refine_advance_kernel(unsigned* P, int it, const int* count, const unsigned* rej, int nrej,
                                      int* progress, int nbands) {
    if (threadIdx.x == 0) {
        const unsigned c = (unsigned)*count;
        P[it + 1] = c ? accepted_index(P[it], c - 1, rej, nrej) + 1 : P[it];
    }
    for (int b = threadIdx.x; b < nbands; b += blockDim.x) progress[b] = 0;
}

// Left and right images packed per pixel for the refiner: census (32 bits, or 64 in two words) and
// gray | gx << 8 | gy << 16, so a candidate's cost needs one load of each side.
template <bool C64>
struct RPack;
template <>
struct __align__(8) RPack<false> {
    uint32_t c, g;
};
template <>
struct __align__(16) RPack<true> {
    unsigned long long c;
    uint32_t g, pad;
};

template <bool C64>
__global__ void refine_pack_kernel(CostCtx c, RPack<C64>* __restrict__ lp, RPack<C64>* __restrict__ rp) {
    const int n = c.w * c.h;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        RPack<C64> a, b;
        if constexpr (C64) {
            a.c = c.cl64[i];
            b.c = c.cr64[i];
            a.pad = b.pad = 0;
        } else {
            a.c = c.cl[i];
            b.c = c.cr[i];
        }
        a.g = (uint32_t)c.lgray[i] | ((uint32_t)c.lgx[i] << 8) | ((uint32_t)c.lgy[i] << 16);
        b.g = (uint32_t)c.rgray[i] | ((uint32_t)c.rgx[i] << 8) | ((uint32_t)c.rgy[i] << 16);
        lp[i] = a;
        rp[i] = b;
    }
}

// The refiner's local cost, local_cost (src/refiner.cpp:14-36), from packed pixels: the same LUT
// terms added in the same order.
template <bool C64>
__device__ __forceinline__ float packed_cost(const CostCtx& c, const float* lut, const RPack<C64>& l,
                                             const RPack<C64>& r) {
    int pop;
    if constexpr (C64) pop = __popcll(l.c ^ r.c);
    else pop = __popc(l.c ^ r.c);
    float v = lut[kLutCensus + pop];
    const uint32_t dd = __vabsdiffu4(l.g, r.g);  // |dgray|, |dgx|, |dgy|
    if (c.use_ad) v = __fadd_rn(v, lut[kLutAd + (dd & 0xFFu)]);
    if (c.use_grad) v = __fadd_rn(v, lut[kLutGrad + ((dd >> 8) & 0xFFu) + (dd >> 16)]);
    return v;
}

// Everything about one pixel of a pass that does not depend on the wavefront, computed for all
// pixels at once before the pass and laid out in wavefront order: its range and the two static
// candidates -- the current value and the current value plus the pixel's draw -- with their
// costs.  The band kernel only costs the two dynamic candidates (left and up neighbours) and keeps
// the reference's candidate order.  A pixel the pass does not update carries the cost -infinity and
// its value as a neighbour candidate (roundf(value) when value >= 0, else -1), so the same selection
// returns it; an updated pixel without a value carries the cost 1e9 and the start of its range.
// The pixel's packed left image rides along.
template <bool C64>
struct __align__(16) RStep {
    float c_cur;   // cost of candidate d_cur
    float c_draw;  // cost of candidate d_draw (1e9: none)
    int lo, hi1;   // the range's first and last disparity
    int d_cur, d_draw;
    RPack<C64> left;
};
static_assert(sizeof(RStep<false>) == 32 && sizeof(RStep<true>) == 48, "bulk copies of whole records");

template <bool C64>
__device__ __forceinline__ float cand_cost(const CostCtx& c, const float* lut, const RPack<C64>& l,
                                           const RPack<C64>* __restrict__ rp, int x, int y, int d, int lo, int hi) {
    const int xr = x - d;
    if (xr >= 0 && xr < c.w && d >= lo && d < hi) return packed_cost<C64>(c, lut, l, rp[y * c.w + xr]);
    return 1e6f;
}

// A value as a neighbour candidate: rounded when it is non-negative, else none (-1).
__device__ __forceinline__ int neighbour(float v) { return v >= 0.f ? (int)roundf(v) : -1; }

// Wavefront order: the records and right-image pixels of a band's step lie together, lane
// by lane ([band][step][lane]), so a chunk of steps is one contiguous bulk copy each.  The right pixels
// start wave_lead(D) steps before the first step: the window of the first columns.
__host__ __device__ inline int wave_chunks(int w) { return (w + kBand - 1 + kChunk - 1) / kChunk; }
__host__ __device__ inline int wave_lead(int D) { return (D - 1 + kChunk - 1) / kChunk * kChunk; }

// A window pixel outside the image: its byte 3 against a left pixel's 0 takes the gradient index past
// kGradIn, where the table holds 1e30.
constexpr uint32_t kOutside = 0xFF000000u;
constexpr uint32_t kGradWeights = 0x03010100u;  // index = |dgx| + |dgy| + 3 * byte 3
constexpr int kGradIn = 511, kGradAll = 3 * 255 + kGradIn;

// A run of a pass's columns: cols of them from column begin, in pass order.
struct ColRun {
    int begin, cols;
};

// One pixel record per (band, step, lane), neutral where the lane has no pixel of the run at that step, and
// the right-image pixel that enters its window at that step (column u of a row brings image column
// x(u) - eoff).  Columns u count from the run's first; the neutral record of column -1 hands the lane the
// candidate that the run before left there.
template <bool C64, bool WIN>
__global__ void __launch_bounds__(256) refine_prep_kernel(CostCtx c, int fwd, ColRun run, const uint8_t* __restrict__ reliable,
                                   const int* __restrict__ prefix, const int16_t* __restrict__ draw_value,
                                   const unsigned* __restrict__ rej, int nrej, const unsigned* __restrict__ P_ptr,
                                   const RPack<C64>* __restrict__ lp, const RPack<C64>* __restrict__ rp,
                                   const float* __restrict__ work, RStep<C64>* __restrict__ steps,
                                   RPack<C64>* __restrict__ wr) {
    __shared__ float s_lut[kLutSize];
    for (int i = threadIdx.x; i < kLutSize; i += blockDim.x) s_lut[i] = c.lut[i];
    __syncthreads();
    const int w = c.w, h = c.h, n = w * h;
    const unsigned P = *P_ptr;
    const int lead = WIN ? wave_lead(c.D) : 0, nstep = wave_chunks(run.cols) * kChunk, tt = lead + nstep;
    const int nbands = (h + kBand - 1) / kBand;
    const int eoff = fwd ? c.d0 : c.d0 + c.D - 1;
    const int lane = threadIdx.x & 31, per = blockDim.x >> 5;
    for (int j = blockIdx.x * per + (threadIdx.x >> 5); j < nbands * tt; j += gridDim.x * per) {
        const int band = j / tt, t = j - band * tt - lead;
        const int v = band * kBand + lane, u = t - lane;
        const int x = fwd ? run.begin + u : w - 1 - run.begin - u;
        const int y = fwd ? v : h - 1 - v;
        if constexpr (WIN) {
            const int pe = x - eoff;
            RPack<C64> e = {};
            e.g = kOutside;
            if (v < h && (unsigned)pe < (unsigned)w) e = rp[(size_t)y * w + pe];
            wr[(size_t)j * 32 + lane] = e;
            if (t < 0) continue;
        }
        RStep<C64> st = {};
        st.c_cur = __int_as_float(0xff800000);
        st.c_draw = 1e9f;
        st.d_cur = -1;
        if (v < h && u == -1 && run.begin > 0) st.d_cur = neighbour(work[y * w + x]);
        if (v < h && (unsigned)u < (unsigned)run.cols) {
            const int i = y * w + x;
            const float cur = work[i];
            const int lo = c.rmin[i], hi = c.rmax[i];
            st.left = lp[i];
            st.lo = lo;
            st.hi1 = hi - 1;
            if (reliable[i] || hi <= lo) {
                st.d_cur = neighbour(cur);
            } else if (cur >= 0.f) {
                st.d_cur = min(max((int)roundf(cur), lo), hi - 1);
                st.c_cur = cand_cost<C64>(c, s_lut, st.left, rp, x, y, st.d_cur, lo, hi);
                const unsigned q = (unsigned)prefix[fwd ? i : n - 1 - i];
                const float dv = __fadd_rn(cur, (float)draw_value[accepted_index(P, q, rej, nrej)]);
                if (dv >= 0.f) {
                    st.d_draw = min(max((int)roundf(dv), lo), hi - 1);
                    st.c_draw = cand_cost<C64>(c, s_lut, st.left, rp, x, y, st.d_draw, lo, hi);
                }
            } else {
                st.c_cur = 1e9f;
                st.d_cur = lo;
            }
        }
        steps[((size_t)band * nstep + t) * 32 + lane] = st;
    }
}

constexpr int kRing = 4 * kChunk;       // steps of pixel records in flight, at most
constexpr int kAhead = 64;              // steps ahead the right-image window is prefetched into L1

__device__ __forceinline__ void prefetch_l1(const void* p) {
    asm volatile("prefetch.global.L1 [%0];\n" ::"l"(p));
}

// Progress counters between bands use the fence forms of release and acquire: the publishing lane
// fences (acquire-release, device scope) and then stores the counter; the reading band polls the
// counter and fences before reading the row above.
__device__ __forceinline__ void fence_acq_rel() { asm volatile("fence.acq_rel.gpu;\n" ::: "memory"); }

// The row above a band, as neighbour candidates (roundf(value) when value >= 0, else -1): column u at
// up[u + kUpShift], with one single-use mbarrier per kChunk positions.  The shift puts the columns a
// band's last lane finishes in one chunk (column t - 31 at step t) on one barrier and one 32-byte line.
constexpr int kUpShift = (kBand - 1) % kChunk;
__host__ __device__ inline int up_blocks(int w) { return (w + kUpShift - 1) / kChunk + 1; }

// Shared state between the compute warp (warp 0) and the link warp (warp 1) of a band at the edge of a
// cluster.  Inside a cluster a band's compute warp sends its last row straight into the next band's
// shared memory (st.async, which completes on the receiver's barriers).  Between clusters the link warps
// carry the exchange, so that no GPU-scope fence or L2 round trip sits in the compute warp's steps:
//   * the link warp of a cluster's first band polls the band above's progress counter, copies the newly
//     final columns of that band's last row into `up` and arrives on their barriers;
//   * that of a cluster's last band publishes how far the last row is final (`done`, raised by the
//     compute warp at CTA scope) to the band's progress counter, behind a GPU-scope fence.
struct BandLink {
    int done;   // columns [0, done) of the band's last row are final in `work` (compute warp)
    int abort;  // the link warp gave up waiting (or saw the error word): the compute warp stops
};

// ---- the band kernel's step ring: mbarriers between the loader warp and the compute warp
__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* b, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n}\n" ::"r"(smem_u32(b)) : "memory");
}
__device__ __forceinline__ bool mbar_done(uint64_t* b, unsigned parity) {
    unsigned ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(ok)
                 : "r"(smem_u32(b)), "r"(parity)
                 : "memory");
    return ok != 0;
}
// Waits, in every lane of the warp, for the completed phase `parity` of b; the warp leaves the
// wait together.  False after `limit` polls (each followed by a sleep of `sleep_ns` when non-zero)
// or once *stop is raised.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* b, unsigned parity, int limit, const volatile int* stop,
                                               int sleep_ns) {
    for (int spins = 0;; ++spins) {
        if (__all_sync(0xffffffffu, mbar_done(b, parity))) return true;
        if (spins >= limit || (stop && *stop)) return false;
        if (sleep_ns) __nanosleep(sleep_ns);
    }
}

__device__ __forceinline__ void mbar_expect(uint64_t* b, unsigned bytes) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n}\n" ::"r"(smem_u32(b)), "r"(bytes)
                 : "memory");
}
// contiguous copy of this GPU's global memory to shared memory, completing on b (16-byte multiples)
__device__ __forceinline__ void bulk_load(void* dst, const void* src, unsigned bytes, uint64_t* b) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(b))
                 : "memory");
}
// the same shared-memory address in CTA `rank` of the cluster
__device__ __forceinline__ unsigned peer_smem(unsigned addr, unsigned rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_async4(unsigned addr, int a, int b, int c, int d, unsigned bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];\n" ::"r"(addr),
                 "r"(a), "r"(b), "r"(c), "r"(d), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;\n" ::: "memory");
}

// The link warp of a band that receives from (recv) or publishes to (send) another cluster.  Every wait
// is bounded: after spin_limit polls in which nothing moved it sets the error word and `abort`, and after
// as many again it leaves.
__device__ void band_link(BandLink* s_link, int* s_up, uint64_t* upbar, int band, int width, int h, ColRun run,
                          int fwd, const float* work, int* progress, int* err, int spin_limit, bool recv, bool send) {
    const int lane = threadIdx.x & 31;
    volatile BandLink* L = s_link;
    volatile int* vprog = progress;
    const int w = run.cols;
    const int xs = fwd ? 1 : -1, xb = fwd ? run.begin : width - 1 - run.begin;
    const int y_above = recv ? (fwd ? band * kBand - 1 : h - band * kBand) : 0;
    const float* above = work + (size_t)y_above * width;
    int fetched = recv ? 0 : w;      // columns of the row above copied
    int blocks = 0;                  // barriers arrived on
    int published = send ? 0 : w;
    int idle = 0;
    bool gave_up = false;
    for (;;) {
        bool moved = false;
        // this band's last row, as far as the compute warp has released it
        const int done = L->done;
        if (done > published) {
            if (lane == 0) {
                fence_acq_rel();
                vprog[band] = done;
            }
            published = done;
            moved = true;
        }
        if (published >= w && (fetched >= w || gave_up)) break;
        // the row above, as far as the band above has published it
        if (fetched < w && !gave_up) {
            int prog = 0;
            if (lane == 0) prog = vprog[band - 1];
            prog = min(__shfl_sync(0xffffffffu, prog, 0), w);
            if (prog > fetched) {
                if (lane == 0) fence_acq_rel();
                __syncwarp();
                for (int col = fetched + lane; col < prog; col += 32) {
                    s_up[col + kUpShift] = neighbour(__ldcg(above + (xb + xs * col)));
                }
                __syncwarp();
                fetched = prog;
                const int upto = fetched >= w ? up_blocks(w) : (fetched + kUpShift) / kChunk;
                if (lane == 0) {
                    __threadfence_block();
                    for (int b = blocks; b < upto; ++b) mbar_arrive(&upbar[b]);
                }
                blocks = upto;
                moved = true;
            }
        }
        if (moved) {
            idle = 0;
            continue;
        }
        ++idle;
        if (!gave_up && (idle > spin_limit || *(volatile int*)err)) {
            if (lane == 0) {
                atomicExch(err, 1);
                L->abort = 1;
            }
            gave_up = true;
            idle = 0;
        } else if (gave_up && idle > spin_limit) {
            break;  // the compute warp did not finish either: leave (the frame is already failed)
        }
        __nanosleep(32);
    }
}

// Shared memory of the band kernel besides the row above and the window.
template <bool C64>
struct BandRing {
    static constexpr int kSlots = C64 ? 2 : 4;    // chunks in flight
    static_assert(kSlots * kChunk <= kRing, "the window ring covers the steps copied ahead");
    RStep<C64> rec[kSlots * kChunk][32];          // chunk k's records in slot k % kSlots, one per step and lane
    uint64_t full[kSlots];      // chunk filled (its bulk copies landed)
    uint64_t empty[kSlots];     // chunk read (one arrival of the compute warp)
    int stop;                   // the compute warp has stopped: the loader stops too
};

// The loader warp: bulk copies of a chunk's records and (WIN) the right-image pixels that enter the window, which land on full[slot], up to kSlots chunks ahead of the compute warp, refilling a
// slot only once the compute warp has released it.  Without WIN it keeps the right-image window warm in L1
// instead: every lane misses L1 at a different step and the compute warp waits for the slowest, so the
// window's first kAhead steps are prefetched first and its entering edge kAhead steps ahead of the copies.
template <bool C64, bool WIN>
__device__ void band_loader(const CostCtx& c, int band, ColRun run, int fwd, BandRing<C64>* ring, RPack<C64>* s_win, int wmask,
                            const RStep<C64>* steps, const RPack<C64>* wr, const RPack<C64>* rp, int spin_limit) {
    const int w = c.w, lane = threadIdx.x & 31;
    const int nchunks = wave_chunks(run.cols), nstep = nchunks * kChunk;
    const int lead = WIN ? wave_lead(c.D) : 0;
    const RStep<C64>* gs = steps + (size_t)band * nstep * 32;
    const RPack<C64>* gr = wr + ((size_t)band * (lead + nstep) + lead) * 32;
    constexpr int kSlots = BandRing<C64>::kSlots;
    constexpr unsigned bs = kChunk * 32 * sizeof(RStep<C64>), bp = kChunk * 32 * sizeof(RPack<C64>);
    const int v = band * kBand + lane, y = fwd ? v : c.h - 1 - v;
    const int xs = fwd ? 1 : -1, xb = fwd ? run.begin : w - 1 - run.begin, eoff = fwd ? c.d0 : c.d0 + c.D - 1;
    const RPack<C64>* rrow = rp + (size_t)(v < c.h ? y : 0) * w;
    if (!WIN)
        for (int k = -c.D; k <= kAhead; k += 8) prefetch_l1(rrow + min(max(xb + xs * k - eoff, 0), w - 1));
    int issued = 0;
    for (int k = 0; k < nchunks; ++k) {
        const int slot = k % kSlots;
        if (k >= kSlots &&
            !mbar_wait_warp(&ring->empty[slot], ((k / kSlots) - 1) & 1, spin_limit, &ring->stop, 32))
            break;  // the compute warp stopped, or never released the slot: it fails the pass itself
        if (lane == 0) {
            const unsigned first = WIN && k == 0 ? (unsigned)lead * 32 * (unsigned)sizeof(RPack<C64>) : 0u;
            mbar_expect(&ring->full[slot], bs + (WIN ? bp + first : 0u));
            const size_t o = (size_t)k * kChunk * 32;
            bulk_load(&ring->rec[slot * kChunk][0], gs + o, bs, &ring->full[slot]);
            if (WIN) {
                // the window ring holds step t's entering pixels at t & wmask
                if (first) bulk_load(s_win + (size_t)(wmask + 1 - lead) * 32, gr - (size_t)lead * 32, first, &ring->full[slot]);
                bulk_load(s_win + (size_t)((k * kChunk) & wmask) * 32, gr + o, bp, &ring->full[slot]);
            }
        }
        issued = k + 1;
        if (!WIN) {
#pragma unroll
            for (int i = 0; i < kChunk; ++i)
                prefetch_l1(rrow + min(max(xb + xs * (k * kChunk + i - lane + kAhead) - eoff, 0), w - 1));
        }
        __syncwarp();
    }
    // no copy may land after the block has left: wait for the chunks still in flight
    for (int k = max(0, issued - kSlots); k < issued; ++k)
        mbar_wait_warp(&ring->full[k % kSlots], (k / kSlots) & 1, 1 << 23, nullptr, 0);
}

// packed_cost for the wavefront's steps: one byte-difference instruction for the three differences, every
// table read (the entries of a term the configuration leaves out are zero, and adding zero changes no
// sum), the gradient table extended to kGradAll entries so that a pixel outside the image costs 1e30.
template <bool C64>
__device__ __forceinline__ float step_cost(const float* lut, const RPack<C64>& l, const RPack<C64>& r) {
    int pop;
    if constexpr (C64) pop = __popcll(l.c ^ r.c);
    else pop = __popc(l.c ^ r.c);
    const uint32_t dd = __vabsdiffu4(l.g, r.g);
    return __fadd_rn(__fadd_rn(lut[kLutCensus + pop], lut[kLutAd + (dd & 0xFFu)]),
                     lut[kLutGrad + __dp4a(dd, kGradWeights, 0u)]);
}

// WIN: the lanes' right-image windows ([x - dmax + 1, x - d0] of each row, sliding one pixel per step)
// live in shared memory, a ring of wmask + 1 steps (a power of two holding the window plus the kRing
// steps copied ahead): the pixels entering at step t lie at t & wmask, lane by lane, so a candidate's
// right pixel is a conflict-free shared-memory load a known number of steps back.  Without WIN they are
// global loads kept warm in L1 by the loader's prefetches.  Three warps per block: warp 0 computes,
// warp 1 links the band to other clusters (band_link), warp 2 loads the rings (band_loader).
//
// Bound: the step's dependent chain -- neighbour shuffle, clamp, window load, table loads, two adds,
// four selects -- times about w + 40 bands steps a pass.  Everything else is kept off the step: waits
// and hand-overs come once per chunk of eight steps, the chunk's steps are one straight line of code
// without divergent branches (a pixel that is not updated takes the same selection, see RStep), its
// records come by bulk copies that use no issue slot or load path of the SM, and a band hands its last
// row to the next one through the cluster's shared memory.
template <bool C64, bool WIN, bool FWD>
__global__ void __launch_bounds__(96) refine_band_kernel(CostCtx c, int band0, int nbands, int csize, ColRun run,
                                                         const RStep<C64>* __restrict__ steps,
                                                         const RPack<C64>* __restrict__ wr,
                                                         const RPack<C64>* __restrict__ rp, float* work,
                                                         int* progress, int* err, int spin_limit, int wmask) {
    constexpr int fwd = FWD ? 1 : 0;
    constexpr int kSlots = BandRing<C64>::kSlots;
    __shared__ float s_lut[kLutGrad + kGradAll];
    __shared__ __align__(128) BandRing<C64> s_ring;
    __shared__ BandLink s_link;
    extern __shared__ __align__(128) unsigned char s_dyn[];
    const int w = run.cols;  // columns of the run: everything below but addresses counts in them
    const int ublk = up_blocks(w);
    RPack<C64>* s_win = reinterpret_cast<RPack<C64>*>(s_dyn);
    int* s_up = reinterpret_cast<int*>(s_dyn + (WIN ? (size_t)(wmask + 1) * 32 * sizeof(RPack<C64>) : 0));
    uint64_t* s_upbar = reinterpret_cast<uint64_t*>(s_up + ublk * kChunk);
    const int band = band0 + (int)blockIdx.x;  // a group of bands starts with a cluster
    const int rank = (int)blockIdx.x % csize;
    const bool live = band < nbands;
    // the row above comes from the cluster's previous band, from another cluster, or (band 0) nowhere
    const bool from_peer = live && rank > 0, from_link = live && band > 0 && rank == 0;
    const bool to_peer = live && rank + 1 < csize && band + 1 < nbands;
    const bool to_link = live && rank + 1 == csize && band + 1 < nbands;
    for (int i = threadIdx.x; i < kLutGrad + kGradAll; i += blockDim.x) s_lut[i] = i < kLutGrad + kGradIn ? c.lut[i] : 1e30f;
    for (int i = threadIdx.x; i < ublk; i += blockDim.x) mbar_init(&s_upbar[i], 1);
    if (threadIdx.x == 0) {
        s_link.done = 0;
        s_link.abort = 0;
        s_ring.stop = 0;
        for (int i = 0; i < kSlots; ++i) {
            mbar_init(&s_ring.full[i], 1);
            mbar_init(&s_ring.empty[i], 1);
        }
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    __syncthreads();
    if (from_peer)
        for (int i = threadIdx.x; i < ublk; i += blockDim.x) mbar_expect(&s_upbar[i], kChunk * 4);
    __syncthreads();
    cluster_sync();  // every band's barriers are armed before a peer sends
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    if (live && warp == 1) {
        if (from_link || to_link)
            band_link(&s_link, s_up, s_upbar, band, c.w, c.h, run, fwd, work, progress, err, spin_limit, from_link, to_link);
    } else if (live && warp == 2) {
        band_loader<C64, WIN>(c, band, run, fwd, &s_ring, s_win, wmask, steps, wr, rp, spin_limit);
    } else if (live) {
        volatile BandLink* link = &s_link;
        const int v = band * kBand + lane;
        const int yrow = fwd ? v : c.h - 1 - v;
        const int xs = fwd ? 1 : -1, xb = fwd ? run.begin : c.w - 1 - run.begin;
        const size_t rowoff = (size_t)(v < c.h ? yrow : 0) * c.w;
        float* wrow = work + rowoff;
        const RPack<C64>* rrow = rp + rowoff;
        const unsigned peer_up = to_peer ? peer_smem(smem_u32(s_up), rank + 1) : 0u;
        const unsigned peer_bar = to_peer ? peer_smem(smem_u32(s_upbar), rank + 1) : 0u;
        // steps back to a candidate's window pixel: back_0 + d forward, back_0 - d backward (the entering
        // pixel has the lowest disparity forward, the highest backward)
        const int back_0 = fwd ? -c.d0 : c.d0 + c.D - 1;
        // Neighbour values travel as candidates: roundf(value) when value >= 0, else -1 (the
        // reference takes a neighbour only when it is non-negative, rounded), or any negative value.
        // candidate of this lane's previous column (its left neighbour); the neutral records before a lane's
        // first column set it again
        int prev = run.begin > 0 && v < c.h ? neighbour(wrow[xb - xs]) : -1;
        bool abort = false;
        const int nchunks = wave_chunks(w);
        int upc = band > 0 ? 0 : ublk;  // barriers of the row above known to be complete
        int sent = 0;                   // blocks of this band's last row sent to the peer
        for (int k = 0; k < nchunks && !abort; ++k) {
            const int t0 = k * kChunk;
            // the row above up to column t0 + kChunk - 1 (lane 0's up neighbours)
            const int need = min((t0 + kChunk - 1 + kUpShift) / kChunk + 1, ublk);
            while (upc < need) {
                if (!mbar_wait_warp(&s_upbar[upc], 0, spin_limit, &s_link.abort, 0)) {
                    abort = true;
                    break;
                }
                ++upc;
            }
            // the chunk's slot has landed
            const int slot = k % kSlots;
            if (abort || !mbar_wait_warp(&s_ring.full[slot], (k / kSlots) & 1, spin_limit, nullptr, 0)) {
                abort = true;
                break;
            }
            int up_first[kChunk];
#pragma unroll
            for (int i = 0; i < kChunk; ++i)
                up_first[i] = band > 0 ? s_up[min(t0 + i + kUpShift, ublk * kChunk - 1)] : -1;
            const RStep<C64>* recs = &s_ring.rec[slot * kChunk][lane];
            const int x0 = xb + xs * (t0 - lane);
            int last[kChunk];
#pragma unroll
            for (int i = 0; i < kChunk; ++i) {
                const int up_lane = __shfl_up_sync(0xffffffffu, prev, 1);
                const int up = lane > 0 ? up_lane : up_first[i];
                const RStep<C64> st = recs[i * 32];
                // dynamic candidates: left (forward) / right (backward) and up / down, clamped into the
                // range
                const int dl = min(max(prev, st.lo), st.hi1), du = min(max(up, st.lo), st.hi1);
                RPack<C64> pl, pu;
                if constexpr (WIN) {
                    // byte offsets into the ring, 32 pixels a step
                    constexpr int B = 32 * (int)sizeof(RPack<C64>);
                    const int base = (t0 + i - back_0) * B, m = wmask * B;
                    const unsigned char* win = reinterpret_cast<const unsigned char*>(s_win + lane);
                    pl = *reinterpret_cast<const RPack<C64>*>(win + ((FWD ? base - dl * B : base + dl * B) & m));
                    pu = *reinterpret_cast<const RPack<C64>*>(win + ((FWD ? base - du * B : base + du * B) & m));
                } else {
                    const int xl = x0 + xs * i - dl, xu = x0 + xs * i - du;
                    const bool in_l = (unsigned)xl < (unsigned)c.w, in_u = (unsigned)xu < (unsigned)c.w;
                    pl = rrow[in_l ? xl : 0];
                    pu = rrow[in_u ? xu : 0];
                    pl.g = in_l ? pl.g : kOutside;
                    pu.g = in_u ? pu.g : kOutside;
                }
                // a neighbour outside the image costs 1e6 like the reference's; no neighbour never wins
                const float vl = step_cost<C64>(s_lut, st.left, pl), vu = step_cost<C64>(s_lut, st.left, pu);
                const float il = vl < 1e29f ? vl : 1e6f, iu = vu < 1e29f ? vu : 1e6f;
                const float cl = prev >= 0 ? il : 1e30f, cu = up >= 0 ? iu : 1e30f;
                // the reference's order: cur, left, up, cur + draw; the first strict minimum wins (as two
                // pairs, the second winning only if strictly below the first)
                const int da = cl < st.c_cur ? dl : st.d_cur, db = st.c_draw < cu ? st.d_draw : du;
                const float ca = fminf(cl, st.c_cur), cb = fminf(st.c_draw, cu);
                prev = cb < ca ? db : da;
                if (st.c_cur != __int_as_float(0xff800000)) wrow[x0 + xs * i] = (float)prev;
                last[i] = prev;
            }
            // every lane has read the slot (and its window pixels): the loader may refill it
            __syncwarp();
            if (lane == 0) mbar_arrive(&s_ring.empty[slot]);
            // hand on the last row's columns of this chunk (lane 31, column t - 31)
            if (to_peer) {
                const int pos = t0 - (kBand - 1) + kUpShift;  // a multiple of kChunk
                if (pos >= 0 && pos < ublk * kChunk) {
                    if (lane == kBand - 1) {
                        const unsigned dst = peer_up + pos * 4, bar = peer_bar + pos / kChunk * 8;
                        st_async4(dst, last[0], last[1], last[2], last[3], bar);
                        st_async4(dst + 16, last[4], last[5], last[6], last[7], bar);
                    }
                    sent = pos / kChunk + 1;
                }
            } else if (to_link) {
                __threadfence_block();
                if (lane == kBand - 1) link->done = max(0, min(t0 + kChunk - (kBand - 1), w));
            }
        }
        if (abort) {
            if (lane == 0) atomicExch(err, 1);
            *(volatile int*)&s_ring.stop = 1;
        }
        __syncwarp();
        __threadfence_block();
        // the whole band is final (or the pass was abandoned: let the next band finish).  Every block of
        // the row is sent whatever happened, and every band takes all of its own before it leaves, so no
        // store is under way to a block that has ended.
        if (lane == kBand - 1) {
            link->done = w;
            if (to_peer)
                for (int b = sent; b < ublk; ++b) {
                    st_async4(peer_up + b * (kChunk * 4), -1, -1, -1, -1, peer_bar + b * 8);
                    st_async4(peer_up + b * (kChunk * 4) + 16, -1, -1, -1, -1, peer_bar + b * 8);
                }
        }
        __syncwarp();
        if (from_peer)
            for (; upc < ublk; ++upc) mbar_wait_warp(&s_upbar[upc], 0, 1 << 23, nullptr, 0);
    }
    __syncwarp();
    cluster_sync();  // a peer's last stores have a block to land in
}

// ---- host: the engine stream, its draw values and rejected indices per radius

struct DrawTable {
    std::vector<int16_t> value;
    std::vector<unsigned> rejected;
};

std::mutex g_rng_mu;
std::vector<uint32_t> g_raw;          // std::mt19937(12345) outputs, generated on demand
std::mt19937 g_engine(12345);
std::map<int, DrawTable> g_tables;   // by radius

// A generator that replays recorded engine outputs, counting how many the distribution takes.
struct Replay {
    using result_type = std::mt19937::result_type;
    const uint32_t* p;
    int calls = 0;
    static constexpr result_type min() { return std::mt19937::min(); }
    static constexpr result_type max() { return std::mt19937::max(); }
    result_type operator()() { return p[calls++]; }
};

const DrawTable& draw_table_locked(int radius, size_t length) {
    while (g_raw.size() < length + 64) g_raw.push_back((uint32_t)g_engine());
    DrawTable& t = g_tables[radius];
    std::uniform_int_distribution<int> dist(-radius, radius);
    for (size_t i = t.value.size(); i < length; ++i) {
        Replay g{g_raw.data() + i};
        const int v = dist(g);
        t.value.push_back((int16_t)v);
        if (g.calls != 1) t.rejected.push_back((unsigned)i);  // output i is skipped by the distribution
    }
    return t;
}

}  // namespace

size_t refine_scan_temp_bytes(int n) { return (size_t)((n + 1 + kScanTile - 1) / kScanTile) * sizeof(int); }

int refine_band_count(int h) { return (h + kBand - 1) / kBand; }

int RefineTables::build(int iterations, int base_radius, int n) {
    release();
    std::vector<const DrawTable*> tabs(iterations);
    std::vector<size_t> len(iterations);
    // until the tables are copied: another thread's longer frame moves a table as it grows it
    std::lock_guard<std::mutex> lk(g_rng_mu);
    for (int it = 0; it < iterations; ++it) {
        const int radius = std::max(1, base_radius >> it);
        if (radius > 32767) return 1;
        // pass `it` starts at most it * n outputs (plus rejections) into the stream
        len[it] = (size_t)(it + 1) * n + 64;
        tabs[it] = &draw_table_locked(radius, len[it]);
        if (tabs[it]->rejected.size() > (size_t)kMaxRejected) return 1;
    }
    iters = iterations;
    size_t total = 0;
    for (int it = 0; it < iterations; ++it) total += len[it] * 2 + kMaxRejected * 4 + 256;
    if (cudaMalloc(&dev, total) != cudaSuccess) {
        cudaGetLastError();
        dev = nullptr;
        return 1;
    }
    bytes = total;
    unsigned char* p = static_cast<unsigned char*>(dev);
    for (int it = 0; it < iterations; ++it) {
        const DrawTable& t = *tabs[it];
        value[it] = reinterpret_cast<int16_t*>(p);
        if (copy_in(p, t.value.data(), len[it] * 2) != cudaSuccess) return 1;
        p += (len[it] * 2 + 255) & ~size_t(255);
        rejected[it] = reinterpret_cast<unsigned*>(p);
        size_t nr = 0;
        for (unsigned r : t.rejected)
            if (r < len[it]) ++nr;
        nrej[it] = (int)nr;
        if (nr && copy_in(p, t.rejected.data(), nr * 4) != cudaSuccess) return 1;
        p += kMaxRejected * 4;
    }
    n_built = n;
    radius_built = base_radius;
    return 0;
}

void RefineTables::release() {
    if (dev) cudaFree(dev);
    dev = nullptr;
    bytes = 0;
    iters = 0;
    n_built = 0;
}

cudaError_t launch_refine_count(const Layout& L, unsigned char* arena, const float* work, int fwd,
                                cudaStream_t s, unsigned* launches) {
    const int n = L.w * L.h;
    int* flags = reinterpret_cast<int*>(arena + L.rf_prefix);
    const int blocks = min((n + 256) / 256, 148 * 8);
    refine_flags_kernel<<<blocks, 256, 0, s>>>(L.w, L.h, reinterpret_cast<const uint8_t*>(arena + L.reliable),
                                                reinterpret_cast<const int16_t*>(arena + L.rmin),
                                                reinterpret_cast<const int16_t*>(arena + L.rmax), work, fwd, flags);
    // the draw indices: exclusive prefix sum of the n + 1 flags (the last one 0), in place
    const int m = n + 1;
    const int nt = (m + kScanTile - 1) / kScanTile;
    int* sums = reinterpret_cast<int*>(arena + L.rf_scan_tmp);
    scan_tile_sums_kernel<<<nt, kScanThreads, 0, s>>>(flags, m, sums);
    scan_tile_offsets_kernel<<<1, kScanThreads, 0, s>>>(sums, nt);
    scan_apply_kernel<<<nt, kScanThreads, 0, s>>>(flags, m, sums);
    *launches += 4;
    return cudaGetLastError();
}

cudaError_t launch_refine_pack(const CostCtx& c, const Layout& L, unsigned char* arena, cudaStream_t s,
                               unsigned* launches) {
    const int n = L.w * L.h;
    const int blocks = min((n + 255) / 256, 148 * 8);
    if (c.census64)
        refine_pack_kernel<true><<<blocks, 256, 0, s>>>(c, reinterpret_cast<RPack<true>*>(arena + L.rf_pack),
                                                        reinterpret_cast<RPack<true>*>(arena + L.rf_pack) + n);
    else
        refine_pack_kernel<false><<<blocks, 256, 0, s>>>(c, reinterpret_cast<RPack<false>*>(arena + L.rf_pack),
                                                         reinterpret_cast<RPack<false>*>(arena + L.rf_pack) + n);
    ++*launches;
    return cudaGetLastError();
}

size_t refine_pack_bytes(int n, bool c64) { return (size_t)n * 2 * (c64 ? sizeof(RPack<true>) : sizeof(RPack<false>)); }

size_t refine_steps_bytes(int w, int h, int D, bool c64) {
    const size_t nb = refine_band_count(h), nstep = (size_t)wave_chunks(w) * kChunk;
    const size_t pk = c64 ? sizeof(RPack<true>) : sizeof(RPack<false>);
    return nb * 32 * (nstep * (c64 ? sizeof(RStep<true>) : sizeof(RStep<false>)) + (c64 ? 0 : (nstep + wave_lead(D)) * pk));
}

namespace {

// How a pass runs: in clusters of `csize` bands, `cols` columns and up to `group` bands (whole clusters) a
// launch, `smem` bytes and a window ring of wmask + 1 steps a block (csize 0: not at all).
struct PassPlan {
    int csize, group, cols, wmask;
    size_t smem;
};

template <bool C64, bool WIN>
cudaError_t launch_pass_t(const CostCtx& c, const Layout& L, unsigned char* arena, const RefineTables& tab, int it,
                          float* work, int spin_limit, const PassPlan& plan, cudaStream_t s, unsigned* launches) {
    const int fwd = (it % 2) == 0;
    const int n = L.w * L.h;
    const int nbands = refine_band_count(L.h);
    const uint8_t* rel = reinterpret_cast<const uint8_t*>(arena + L.reliable);
    const int* prefix = reinterpret_cast<const int*>(arena + L.rf_prefix);
    unsigned* P = reinterpret_cast<unsigned*>(arena + L.rf_state);
    int* err = reinterpret_cast<int*>(arena + L.rf_state) + kRefineErrWord;
    int* progress = reinterpret_cast<int*>(arena + L.rf_state) + kRefineProgWord;
    const RPack<C64>* lpk = reinterpret_cast<const RPack<C64>*>(arena + L.rf_pack);
    const RPack<C64>* rpk = lpk + n;
    RStep<C64>* steps = reinterpret_cast<RStep<C64>*>(arena + L.rf_steps);
    for (int begin = 0; begin < L.w; begin += plan.cols) {
        const ColRun run{begin, std::min(plan.cols, L.w - begin)};
        const size_t ns = (size_t)nbands * wave_chunks(run.cols) * kChunk * 32;
        RPack<C64>* wr = reinterpret_cast<RPack<C64>*>(steps + ns);
        const size_t items = ns / 32 + (WIN ? (size_t)nbands * wave_lead(c.D) : 0);
        const int blocks = (int)std::min<size_t>((items + 7) / 8, 148 * 8);
        refine_prep_kernel<C64, WIN><<<blocks, 256, 0, s>>>(c, fwd, run, rel, prefix, tab.value[it], tab.rejected[it],
                                                            tab.nrej[it], P + it, lpk, rpk, work, steps, wr);
        ++*launches;
        cudaError_t e = cudaGetLastError();
        // the bands' progress counts a run's columns; refine_advance clears it behind the last run
        if (e == cudaSuccess && begin > 0) e = cudaMemsetAsync(progress, 0, (size_t)nbands * 4, s);
        if (e != cudaSuccess) return e;
        for (int b0 = 0; b0 < nbands; b0 += plan.group) {
            // every band of the group at once (a band waits for the one above): a cooperative launch in clusters
            const int nb = std::min(plan.group, nbands - b0);
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3((nb + plan.csize - 1) / plan.csize * plan.csize);
            cfg.blockDim = dim3(3 * kBand);
            cfg.dynamicSmemBytes = plan.smem;
            cfg.stream = s;
            cudaLaunchAttribute at[2];
            at[0].id = cudaLaunchAttributeCooperative;
            at[0].val.cooperative = 1;
            at[1].id = cudaLaunchAttributeClusterDimension;
            at[1].val.clusterDim.x = plan.csize;
            at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
            cfg.attrs = at;
            cfg.numAttrs = 2;
            e = cudaLaunchKernelEx(&cfg, fwd ? refine_band_kernel<C64, WIN, true> : refine_band_kernel<C64, WIN, false>, c,
                                   b0, nbands, plan.csize, run, (const RStep<C64>*)steps, (const RPack<C64>*)wr, rpk,
                                   work, progress, err, spin_limit, plan.wmask);
            if (e != cudaSuccess) return e;
            ++*launches;
        }
    }
    // start of the next pass, and cleared progress counters
    refine_advance_kernel<<<1, 64, 0, s>>>(P, it, prefix + n, tab.rejected[it], tab.nrej[it], progress, nbands);
    ++*launches;
    return cudaGetLastError();
}

// Sets plan's cluster and group for blocks of plan.smem bytes: the largest cluster (8, 4, 2, 1 bands) in which
// every band of the frame is resident at once; with `parts`, else the largest that fits at all and as many bands
// as are.
template <bool C64, bool WIN, bool FWD>
bool place_bands(int nbands, bool parts, PassPlan& plan) {
    auto kern = refine_band_kernel<C64, WIN, FWD>;
    plan.csize = 0;
    if (allow_dynamic_smem(kern, plan.smem) == cudaSuccess) {
        for (int cs = 8; cs >= 1; cs >>= 1) {
            if (cs > 1 && cs > nbands) continue;
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3((nbands + cs - 1) / cs * cs);
            cfg.blockDim = dim3(3 * kBand);
            cfg.dynamicSmemBytes = plan.smem;
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = cs;
            at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            int nc = 0;
            if (cudaOccupancyMaxActiveClusters(&nc, kern, &cfg) != cudaSuccess) nc = 0;
            if (nc * cs >= (int)cfg.gridDim.x || (parts && nc > 0)) {
                plan.csize = cs;
                plan.group = nc * cs;
                return true;
            }
        }
    }
    cudaGetLastError();
    return false;
}
template <bool C64, bool WIN>
bool place_bands(bool fwd, int nbands, bool parts, PassPlan& plan) {
    return fwd ? place_bands<C64, WIN, true>(nbands, parts, plan) : place_bands<C64, WIN, false>(nbands, parts, plan);
}

}  // namespace

cudaError_t launch_refine_pass(const CostCtx& c, const Layout& L, unsigned char* arena, const RefineTables& tab,
                               int it, float* work, const RefineTuning& tune, cudaStream_t s, unsigned* launches) {
    const int nbands = refine_band_count(L.h);
    const bool fwd = (it % 2) == 0;
    // about a second of waiting at most per wait, unless the engine's tuning sets a smaller poll budget
    const int spin_limit = tune.spin_limit > 0 ? tune.spin_limit : 1 << 23;
    // the right-image window in shared memory (32-bit census): a power-of-two ring of steps holding the
    // window (rounded up to whole chunks) plus the kRing steps copied ahead
    int rs = 1;
    while (rs < wave_lead(c.D) + kRing + kChunk) rs <<= 1;
    const bool win = !c.census64 && tune.window == 0 && rs <= 512;
    PassPlan plan{};
    const auto bare = [&](bool parts) {  // without the window
        plan.wmask = 0;
        plan.smem = (size_t)up_blocks(plan.cols) * (kChunk * 4 + 8);
        return c.census64 ? place_bands<true, false>(fwd, nbands, parts, plan)
                          : place_bands<false, false>(fwd, nbands, parts, plan);
    };
    const auto run_bare = [&] {
        return c.census64 ? launch_pass_t<true, false>(c, L, arena, tab, it, work, spin_limit, plan, s, launches)
                          : launch_pass_t<false, false>(c, L, arena, tab, it, work, spin_limit, plan, s, launches);
    };
    // whole rows where every band of the frame is resident at once with the row above in its block, with the
    // window beside it if that fits too; else in the fewest runs of columns in which they are
    for (int runs = 1;; runs *= 2) {
        plan.cols = (L.w + runs - 1) / runs;
        if (win) {
            plan.wmask = rs - 1;
            plan.smem = (size_t)up_blocks(plan.cols) * (kChunk * 4 + 8) + (size_t)rs * 32 * sizeof(RPack<false>);
            if (place_bands<false, true>(fwd, nbands, false, plan))
                return launch_pass_t<false, true>(c, L, arena, tab, it, work, spin_limit, plan, s, launches);
        }
        if (bare(false)) return run_bare();
        if (plan.cols <= 8 * kBand) break;
    }
    // more bands than any run of columns leaves room for: groups of bands, in the fewest runs that a block holds
    for (int runs = 1;; runs *= 2) {
        plan.cols = (L.w + runs - 1) / runs;
        if (bare(true)) return run_bare();
        if (plan.cols <= 8 * kBand) return cudaErrorCooperativeLaunchTooLarge;
    }
}

}  // namespace apgcu
