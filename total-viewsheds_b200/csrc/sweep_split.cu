// sweep_split.cu -- the direction-split persistent sweep (layouts 1-9).
//
// The reference kernel (kernel.rs:153-254) walks one band of sight and keeps
// the running maximum of angle = (h - h_pov)/d - d/R; a sample is visible
// when its angle is above the maximum, visible samples add d*tan(1 deg) to
// the band's surface and changes of visibility are ring events.
//
// Mapping.  A work item is one warp tile of one sector in one direction: a
// warp holds LX columns x 32/LX rows of lanes and each lane four points of
// view (chains), so a warp's 128 chains cover a compact patch.  Per step the
// chains of a lane share one table entry and one address (in the quad layout
// one 16-byte load gives all four samples).
//
// Scheduling.  The grid is the resident capacity of the GPU.  CTAs take chunks
// of up to kSplitChunk tiles of one (sector, direction) from a global counter
// in sector-major order; the warps of a CTA take the chunk's tiles one by one
// and go on to the next chunk without waiting for each other: a ring of two or
// three chunks with their step tables sits in shared memory, and the warp that
// takes a chunk's last tile brings in the next chunk.  Segment skipping makes the
// tiles' work uneven; with a barrier after every 8 tiles, as before, warps waited
// for the slowest of their CTA and small DEMs for each other (301^2 exact f32:
// 0.94 ms a sweep, now 0.18).
//
// Order.  Every point's surfaces are added sector by sector, forward before
// backward (kernel.rs:254).  An item writes its surfaces to a plane of its own
// (one per sector and direction of the launch; a launch takes as many sectors as
// kPlaneBytes hold), and the last item of a tile adds the planes up in order.  So
// no item waits, and only that last one needs an acquiring fence, which empties
// the SM's L1.  (When every item added its surfaces in turn, behind a fence and
// a wait for the tile's previous item, 37-48 % of the sectors hit L1 in place of
// 72 %, and at 1201^2, where several sectors are under way at once, warps spent
// half their time waiting.)  That way remains for a launch without planes (no
// memory for them, or the failure test's held tile): a counter per tile, and a
// bounded wait.
//
// Arithmetic.  Every step first forms the FP32 estimate of the angle from
// the step's tables, a^ = e*y - c (y = RN(1/d), c = RN(d/R)), with a per-step
// window G above the estimate's error bound (apart from its part relative to
// |a|, which the chain's window carries):
//  * FP32 (the comparison form): the estimate is the angle, fma(e, y, -c).
//  * EXACT32: the running maximum is held exactly; fma(e, y, -c + G) < lo
//    proves that a sample is not visible, and where a chain of the warp passes
//    that test the reference's own f32 angle is evaluated (Markstein division
//    from the table reciprocal).
//  * MIXED64: each chain keeps the estimate mid of its running maximum, the half
//    width hw of the band around it and the step j of the maximum.  f < mid - hw
//    proves the sample is not visible, f > mid + hw that it is.  Only between the
//    two is the comparison re-decided in FP64, against the exact maximum
//    recomputed from step j.
//  * FP64: the running maximum is held in double; where the MIXED64 estimate,
//    raised by its bound, does not prove every chain's sample below the maximum,
//    the angles are evaluated in double.
// So every decision is the exact one, and surfaces add the reference's
// w = RN(d*tan1) in f32 (EXACT32) or RN64(d*0.0174533) in double (MIXED64) in
// step order: bit for bit the reference f32 sweep and the all-FP64 sweep.
// A warp skips a step when no chain can change state (the vote on the first
// test), and a 32-step segment when the DEM's 16x16 block maxima over the
// warp's patch, moved by the segment's offsets, bound every sample below
// every chain's threshold.
//
// Ring records (kRings): chains keep their previous visibility and record
// count; an event (visibility changed) stores the sample's DEM id in the
// band's next slot, slot 1 is the point of view, slot 0 the count at the end
// (kernel.rs:141-145,220-243).  Where a step or a segment is skipped, the chains
// visible before it close their rings at it.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <map>
#include <mutex>
#include <type_traits>
#include <utility>

#include "tvs.h"
#include "tvs_internal.cuh"
#include "queue_sched.cuh"

namespace tvs {
namespace {

constexpr int K = kSplitCols;     // chains per lane
// Iterations of a wait for a chunk of the CTA's own ring (of about 100 ns: seconds,
// against a real wait of at most a few work items).
constexpr uint32_t kRingSpinLimit = 1u << 25;

__device__ __forceinline__ float div_table32(float e, float y, float d) {
    const float q = __fmul_rn(e, y);
    const float r = __fmaf_rn(-d, q, e);
    return __fmaf_rn(r, y, q);
}

__device__ __forceinline__ double div_table64(double e, double y, double d) {
    const double q = __dmul_rn(e, y);
    const double r = __fma_rn(-d, q, e);
    return __fma_rn(r, y, q);
}

// Pairs of floats in one 64-bit register: sm_100's add.f32x2 rounds each half as
// the scalar instruction does and takes one issue slot.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pk(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void upk(f32x2 v, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// MIXED64's guard band.  A sample's estimate f and the maximum's estimate mid (f at
// the step j of the maximum) decide a comparison when they differ by more than
//   hw = 2^-20 |mid| + W_j,   W_j = G_j + the largest G of the steps from j on,
// where G is a step's bound on |f - angle| apart from its part relative to the
// angle.  e = RN(h - h_pov), and the observer height o sits in the step's offset
// z = -(d/R + o/d), so that no rounding is relative to the elevations themselves:
// |f - a| <= 2^-24 (3 |a| + 5 d/R + 6 |o|/d) from the roundings of e, 1/d, z and
// the fma, and the FP64 angle adds 2^-53 (hmax/d + ...).  G = 2^-20 (d/R + |o|/d) +
// 2^-44 hmax/d + 2^-90 holds 2.6 x the absolute part, 2^-20 |mid| the 3 |a| of the
// maximum and of a sample near it 2.6 x; the rounding of f - mid is 2^-24 of a
// value that matters only near hw.  A NaN estimate decides nothing and is not
// visible, as a > m is false for a NaN angle.  (With h_pov + o rounded to f32
// first, the band was 2^-20 hmax/d: on the sea of a 3601^2 tile with 4500 m peaks
// every sample past 330 cells fell into it and was re-decided, 7.6e-4 of all.)
constexpr float kRel = 0x1p-20f;
__device__ __forceinline__ float band_mix(float y, float c, float o, float hmax) {
    return __fadd_rn(__fadd_rn(__fmul_rn(0x1p-20f, __fadd_rn(c, __fmul_rn(fabsf(o), y))),
                               __fmul_rn(0x1p-44f, __fmul_rn(hmax, y))),
                     0x1p-90f);
}
// EXACT32's first test fma(e, y, -d/R + G) >= m - 2^-19 |m| passes every step where
// a chain may change state: e is the reference's own RN(h - RN(h_pov + o)), and
// |e y - d/R - a| <= 2^-24 (4 |a| + 3 d/R) from the roundings of 1/d, the fma and
// the reference's division and subtraction.
constexpr float kRelExact = 0x1p-19f;
__device__ __forceinline__ float window_exact(float c) { return __fmaf_rn(0x1p-20f, c, 0x1p-90f); }

// A step's entry of the table in shared memory: step i's constants are in entry
// i + kAhead, and entry i holds where step i's samples are (next: of the step
// kAhead steps later; the point of view itself past the last step), in floats of
// the DEM or bytes of the quad copies.  One 16-byte read so gives a step its
// constants and the address of the loads that run ahead: two steps for the
// surfaces, one for ring output, whose loop then has one copy of its long body
// (with three, half of its issue slots waited for instructions).
constexpr uint32_t kAheadMost = 2;
template <int kPrec> struct Step;
template <> struct __align__(16) Step<TVS_PRECISION_EXACT32> {
    float y, z, w;  // 1/d, -d/R + G, the surface addend
    int next;
    float d, c;     // the exact angle's d and d/R
    int orig;       // the sample's offset in the DEM (ring ids)
    float pad;
};
template <> struct __align__(16) Step<TVS_PRECISION_MIXED64> {
    float y, z, band;  // 1/d, -(d/R + o/d), W
    int next;
    double w;  // RN64(d*0.0174533)
    int orig;  // the sample's offset in the DEM (ring ids)
    float pad;
};
template <> struct __align__(16) Step<TVS_PRECISION_FP64> {
    float y, z, d;  // 1/d, -(d/R + o/d) + G, d
    int next;
    double y64, c64;  // RN64(1/d), RN64(d/R)
};
template <> struct __align__(16) Step<TVS_PRECISION_FP32> {
    float y, z, w;  // 1/d, -d/R, the surface addend
    int next;
};
template <int kPrec>
using Surface = typename std::conditional<kPrec == TVS_PRECISION_MIXED64 || kPrec == TVS_PRECISION_FP64,
                                          double, float>::type;

// A segment's bounds in this direction: the range of the offsets and the
// extremes of 1/d and of the first test's offset.
struct __align__(16) SegBound {
    int x0, x1, y0, y1;
    float ymax, ymin, zmax, pad;
};

struct SplitSlot {
    QueueDem dem;          // the chunk's DEM (copied from the descriptor array)
    uint32_t group;        // 2 * sector of the launch + direction
    uint32_t tile0, n_tiles;
    uint32_t next;         // next tile of the chunk
    uint32_t left;         // warps that have gone on to the next chunk
    uint32_t end;          // the queue is empty: no chunk
    uint32_t n, n_fast;    // steps, and steps of the table-division loop
    int32_t status;        // the sector's shape status
    uint32_t plain;        // quad layout: the sector reads the plain DEM
};

struct SplitCtl {
    uint32_t ready;              // slots brought in so far
    uint32_t item, upto;         // chunks taken from the queue and not yet in a slot
    unsigned long long diag[4];  // counters, flushed at the end
};

// Shared memory of one CTA: the control block, then the slots of {chunk, step
// table, segment bounds}.
__host__ __device__ constexpr size_t align16(size_t n) { return (n + 15) & ~(size_t)15; }

template <int kPrec> struct SplitSmem {
    __host__ __device__ static size_t slots() { return align16(sizeof(SplitCtl)); }
    __host__ __device__ static size_t table() { return align16(sizeof(SplitSlot)); }
    __host__ __device__ static size_t seg(uint32_t cap) {
        return table() + (size_t)(cap + kAheadMost) * sizeof(Step<kPrec>);
    }
    __host__ __device__ static size_t slot(uint32_t cap) {
        return seg(cap) + (size_t)seg_count(cap) * sizeof(SegBound);
    }
    __host__ __device__ static size_t total(uint32_t cap, uint32_t n_slots) {
        return slots() + n_slots * slot(cap);
    }
};

// Warps per CTA and CTAs per SM: 32 warps of 64 registers a thread for the surface
// sweeps; ring output and FP64 keep more state (24 warps of 80 registers).  24 warps
// of 80 registers measured slower for the other surfaces (1201^2 exact f32 5.03
// against 4.38 ms): the step loop hides its loads with warps.
template <int kPrec, bool kRings> __host__ __device__ constexpr int split_sm_warps() {
    return kRings || kPrec == TVS_PRECISION_FP64 ? 24 : 32;
}
template <int kPrec, bool kRings> __host__ __device__ constexpr int split_warps() {
    return split_sm_warps<kPrec, kRings>() == 32 ? kSplitWarps : 8;
}
template <int kPrec, bool kRings> __host__ __device__ constexpr int split_min_blocks() {
    return split_sm_warps<kPrec, kRings>() / split_warps<kPrec, kRings>();
}

__device__ __forceinline__ uint32_t ld_acquire(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];"
                 : "=r"(v) : "r"((uint32_t)__cvta_generic_to_shared(p)) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(uint32_t *p, uint32_t v) {
    asm volatile("st.release.cta.shared::cta.u32 [%0], %1;"
                 :: "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t add_release(uint32_t *p, uint32_t v) {
    uint32_t old;
    asm volatile("atom.release.gpu.global.add.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
    return old;
}
__device__ __forceinline__ void red_release(uint32_t *p, uint32_t v) {
    asm volatile("red.release.cta.shared::cta.add.u32 [%0], %1;"
                 :: "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(v) : "memory");
}

// The largest of the lanes' values (a NaN is left out), as one reduction.
__device__ __forceinline__ float warp_max(float v) {
    float r;
    asm("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// A visible sample's state change, spelled with predicates: the compiler would
// turn it into a branch and its reconvergence.  The FP32 form: the surface gains
// w, the maximum moves to the angle (false for a NaN: the maximum stays, as
// f32::max has it).
__device__ __forceinline__ void raise_fp32(float ang, float &m, float &s, float w) {
    asm("{\n\t"
        ".reg .pred p;\n\t"
        "setp.gt.f32 p, %2, %0;\n\t"
        "@p add.rn.f32 %1, %1, %3;\n\t"
        "@p mov.f32 %0, %2;\n\t"
        "}"
        : "+f"(m), "+f"(s)
        : "f"(ang), "f"(w));
}
// EXACT32: also the first test's threshold lo = m - 2^-19 |m|.
__device__ __forceinline__ void raise_exact(float ang, float &m, float &s, float &lo, float w) {
    asm("{\n\t"
        ".reg .pred p;\n\t"
        ".reg .f32 t;\n\t"
        "setp.gt.f32 p, %3, %0;\n\t"
        "abs.f32 t, %3;\n\t"
        "@p add.rn.f32 %1, %1, %4;\n\t"
        "@p fma.rn.f32 %2, t, %5, %3;\n\t"
        "@p mov.f32 %0, %3;\n\t"
        "}"
        : "+f"(m), "+f"(s), "+f"(lo)
        : "f"(ang), "f"(w), "f"(-kRelExact));
}
// MIXED64, where x = f - mid >= -hw: hw = 2^-20 |f| + band, the surface gains w, and
// j's half kHi becomes step.  The surface takes w times 1.0 or 0.0 in one rounding
// (the same sum; w is finite and the surface not negative): a predicated FP64 add
// comes out as two selects, this as one.
template <int kHi>
__device__ __forceinline__ void raise_mix(float x, float f, float band, uint32_t step, double w, float &hw,
                                          uint32_t &j, double &acc) {
    asm("{\n\t"
        ".reg .pred p;\n\t"
        ".reg .f32 a, n;\n\t"
        ".reg .b32 h;\n\t"
        ".reg .f64 v;\n\t"
        "neg.f32 n, %0;\n\t"
        "setp.ge.f32 p, %3, n;\n\t"
        "abs.f32 a, %4;\n\t"
        "@p fma.rn.f32 %0, a, %8, %5;\n\t"
        "selp.b32 h, 0x3ff00000, 0, p;\n\t"
        "mov.b64 v, {0, h};\n\t"
        "fma.rn.f64 %2, %7, v, %2;\n\t"
        "@p prmt.b32 %1, %1, %6, %9;\n\t"
        "}"
        : "+f"(hw), "+r"(j), "+d"(acc)
        : "f"(x), "f"(f), "f"(band), "r"(step), "d"(w), "f"(kRel), "n"(kHi ? 0x5410 : 0x3254));
}

// A value that every lane holds, in a uniform register: the branches and shared
// memory addresses that follow from it need no per-lane registers.
__device__ __forceinline__ uint32_t uni(uint32_t v) { return __reduce_max_sync(0xffffffffu, v); }

// MIXED64's exact decision (kernel.rs:175-190 in double, from the shape stage's
// table): is the angle of the sample h at step i above the one of hj at step j
// (-2000 while j < 0)?  Kept out of line: it runs for about one sample in 10^5 and
// its registers would crowd the loop.
__device__ __forceinline__ double mix_angle(float h, float pov, float observer, const double4 *dtab,
                                            uint32_t i) {
    const double y = __ldg(&dtab[i].x), c = __ldg(&dtab[i].y), d = __ldg(&dtab[i].w);
    const double hp = __dadd_rn((double)pov, (double)observer);
    return __dsub_rn(div_table64(__dsub_rn((double)h, hp), y, d), c);
}
__device__ __noinline__ bool mix_visible(float h, float hj, float pov, float observer,
                                         const double4 *dtab, uint32_t i, int32_t j) {
    const double m = j < 0 ? (double)kMaxAngle : mix_angle(hj, pov, observer, dtab, (uint32_t)j);
    return mix_angle(h, pov, observer, dtab, i) > m;
}
template <int kPrec, int kLayout, bool kRings>
__global__ void __launch_bounds__(32 * split_warps<kPrec, kRings>(), (split_min_blocks<kPrec, kRings>()))
k_sweep_split(QueueArgs a, uint32_t n_slots) {
    constexpr int LX = split_lx(kLayout), KY = split_ky(kLayout), KX = K / KY, LY = 32 / LX;
    // rows between a lane's chains: the quad layout reads four consecutive ones
    constexpr int RS = kLayout == kQuadLayout ? 1 : LY, LS = kLayout == kQuadLayout ? KY : 1;
    constexpr int kWarps = split_warps<kPrec, kRings>();
    constexpr bool kFp32 = kPrec == TVS_PRECISION_FP32;
    constexpr bool kMix = kPrec == TVS_PRECISION_MIXED64;
    constexpr bool kF64 = kPrec == TVS_PRECISION_FP64;
    constexpr bool kWide = kMix || kF64;  // surfaces in double
    constexpr uint32_t kAhead = kRings ? 1 : kAheadMost;
    constexpr bool kQuad = kLayout == kQuadLayout;
    using L = SplitSmem<kPrec>;
    using S = Surface<kPrec>;
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t cap = a.max_step_cap;
    SplitCtl &ctl = *reinterpret_cast<SplitCtl *>(smem);
    const uint32_t slot_bytes = (uint32_t)L::slot(cap);
    auto slot_of = [&](uint32_t c) -> unsigned char * {
        return smem + ((uint32_t)L::slots() + c % n_slots * slot_bytes);
    };
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warp = uni(threadIdx.x >> 5);
    const uint32_t n_items = a.chunks * a.n_sectors * 2;
    if (threadIdx.x < 4) ctl.diag[threadIdx.x] = 0;
    if (threadIdx.x == 0) ctl.ready = ctl.item = ctl.upto = 0;
    __syncthreads();

    // Brings chunk c into its slot (one warp): the next item of the queue and
    // its step tables.
    auto bring = [&](uint32_t c) {
        unsigned char *base = slot_of(c);
        SplitSlot &sl = *reinterpret_cast<SplitSlot *>(base);
        Step<kPrec> *s_t = reinterpret_cast<Step<kPrec> *>(base + L::table());
        SegBound *s_seg = reinterpret_cast<SegBound *>(base + L::seg(cap));
        // this CTA's chunks [item, upto); more from the queue when it has none left
        uint32_t item = uni(ctl.item), upto = uni(ctl.upto);
        __syncwarp();
        if (item == upto) {
            // many at a time while many are left, towards the end two tiles per warp
            // of a slot, in a short launch as few as spread it over the GPU
            constexpr uint32_t kMost = kSplitGrab * kWarps / kSplitWarps / (kF64 ? 2 : 1);
            constexpr uint32_t kLeast = kMost / 4 ? kMost / 4 : 1;
            static_assert(kMost >= kLeast, "every grab takes a chunk");
            const uint32_t left = n_items - min(item, n_items);
            const uint32_t grab = left > 2 * kMost * gridDim.x          ? kMost
                                  : n_items >= 4 * kLeast * gridDim.x ? kLeast
                                                                       : 1u;
            item = 0;
            if (lane == 0) item = atomicAdd(a.queue, grab);
            item = uni(item);
            upto = min(item + grab, max(n_items, item));
        }
        uint32_t taken = 0;  // of them, in this slot
        if (item < n_items) {
            const uint32_t group = item / a.chunks, r = item - group * a.chunks;
            const uint32_t dir = group & 1u, slot = a.first_sector + (group >> 1);
            // the DEM whose chunks hold r (chunk_base ascends)
            uint32_t lo = 0, hi = a.n_dems - 1;
            while (lo < hi) {
                const uint32_t mid = (lo + hi + 1) >> 1;
                if (uni(__ldg(&a.dems[mid].chunk_base)) <= r) lo = mid; else hi = mid - 1;
            }
            const uint32_t *src = reinterpret_cast<const uint32_t *>(a.dems + lo);
            uint32_t *dst = reinterpret_cast<uint32_t *>(&sl.dem);
#pragma unroll
            for (uint32_t q = 0; q < sizeof(QueueDem) / 4; q += 32)
                if (q + lane < sizeof(QueueDem) / 4) dst[q + lane] = __ldg(src + q + lane);
            __syncwarp();
            const QueueDem &D = sl.dem;
            const ShapeHeader *h = D.hdr + slot;
            const uint32_t nf = uni(h->n_fast);
            // surfaces stop at the last step that adds to them
            const uint32_t n = uni(kRings ? h->n_steps : max(nf, min(h->n_surf, h->n_steps)));
            const bool wide = uni(h->wide) != 0, plain = !kQuad || wide;
            const float4 *gs = D.steps + (uint64_t)slot * D.step_cap;
            const int2 *go = D.offs + (uint64_t)slot * D.step_cap;
            const int2 *gq = D.quads + (uint64_t)slot * D.step_cap;
            const int4 *gseg = D.segs + (uint64_t)slot * seg_count(D.step_cap);
            const double4 *gd = D.dtab + (uint64_t)slot * D.step_cap;
            (void)gd;
            const float hmax = kWide ? *D.hmax : 0.0f;
            // from the last 32 steps to the first: the band needs the largest G of
            // the later steps
            float later = 0.0f;
            for (uint32_t b = seg_count(n); b-- > 0;) {
                const uint32_t i0 = b * kSegSteps, i = i0 + lane;
                const bool v = i < n;
                float4 t = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                float z = 0.0f, g = 0.0f;
                if (v) {
                    t = gs[i];  // {RN(1/d), d, RN(d/R), RN(d*tan1)}
                    z = -t.z;
                    if constexpr (kWide) {
                        z = -__fadd_rn(t.z, __fmul_rn(D.observer_height, t.x));
                        if (i < nf) g = band_mix(t.x, t.z, D.observer_height, hmax);
                        if constexpr (kF64) z = __fadd_rn(z, g);
                    } else if constexpr (!kFp32) {
                        z = __fadd_rn(z, window_exact(t.z));
                    }
                }
                if constexpr (kMix) {
                    float most = g;  // of this step and the later ones
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const float q = __shfl_down_sync(0xffffffffu, most, o);
                        if (lane + o < 32) most = fmaxf(most, q);
                    }
                    most = fmaxf(most, later);
                    later = __shfl_sync(0xffffffffu, most, 0);
                    g = __fadd_rn(g, most);
                }
                if (v) {
                    int off;
                    if (plain) {
                        off = go[i].x;
                        off = dir ? -off : off;
                    } else {
                        const int2 q = gq[i];
                        off = (dir ? q.y : q.x) * (int)sizeof(float4);
                    }
                    s_t[i].next = off;
                    Step<kPrec> &e = s_t[i + kAhead];
                    e.y = t.x;
                    e.z = z;
                    if constexpr (kRings && !kFp32 && !kF64) e.orig = dir ? -go[i].x : go[i].x;
                    if constexpr (kMix) {
                        e.band = g;
                        e.w = gd[i].z;
                    } else if constexpr (kF64) {
                        e.d = t.y;
                        e.y64 = gd[i].x;
                        e.c64 = gd[i].y;
                    } else {
                        e.w = t.w;
                        if constexpr (!kFp32) {
                            e.d = t.y;
                            e.c = t.z;
                        }
                    }
                }
                if (i0 < nf) {  // these 32 steps are segment b
                    const bool f = i < nf;
                    float ymax = f ? t.x : -INFINITY, ymin = f ? t.x : INFINITY;
                    float zmax = f ? z : -INFINITY;
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) {
                        ymax = fmaxf(ymax, __shfl_xor_sync(0xffffffffu, ymax, o));
                        ymin = fminf(ymin, __shfl_xor_sync(0xffffffffu, ymin, o));
                        zmax = fmaxf(zmax, __shfl_xor_sync(0xffffffffu, zmax, o));
                    }
                    // (no segment of a wide sector is skipped: its linear sample ids wrap into
                    // neighbouring rows, where the moved patch does not bound them)
                    if (wide) zmax = INFINITY;
                    if (lane == 0) {
                        const int4 q = gseg[b];
                        s_seg[b] = dir ? SegBound{-q.y, -q.x, -q.w, -q.z, ymax, ymin, zmax, 0.0f}
                                                    : SegBound{q.x, q.y, q.z, q.w, ymax, ymin, zmax, 0.0f};
                    }
                }
            }
            // the consecutive chunks of this DEM, sector and direction
            const uint32_t tiles = uni(D.tiles_x * D.tiles_y), per = uni(D.chunk);
            const uint32_t tile0 = (r - uni(D.chunk_base)) * per;
            taken = min(upto - item, (tiles - tile0 + per - 1) / per);
            if (lane == 0) {
                for (uint32_t q = 0; q < kAhead; q++) s_t[n + q].next = 0;  // the point of view itself
                sl.tile0 = tile0;
                sl.n_tiles = min(taken * per, tiles - tile0);
                sl.group = group;
                sl.n = n;
                sl.n_fast = nf;
                sl.status = h->status;
                sl.plain = plain;
            }
        }
        __syncwarp();
        if (lane == 0) {
            ctl.item = item + taken;
            ctl.upto = upto;
            sl.next = 0;
            sl.left = 0;
            sl.end = item >= n_items;
            st_release(&ctl.ready, c + 1);
        }
        __syncwarp();
    };
    static_assert(kSegSteps == 32, "a segment's bounds are reduced in one warp, a step per lane");
    // All lanes: waits (bounded) until *p >= v; false: gave up.  The exits are
    // votes, here and below: a loop of one lane would split the warp, and the
    // step loop would then run once for each part.
    auto wait_for = [&](const uint32_t *p, uint32_t v) -> bool {
        uint32_t spins = 0;
        while (!__all_sync(0xffffffffu, ld_acquire(p) >= v)) {
            if (++spins > kRingSpinLimit) {
                if (lane == 0) atomicExch(a.error, (int32_t)TVS_ERR_TIMEOUT);
                __syncwarp();
                return false;
            }
            __nanosleep(100);
        }
        return true;
    };
    // Chunk c can be brought in when every warp has left the chunk whose slot
    // it takes.
    auto slot_free = [&](uint32_t c) -> bool {
        if (c < n_slots) return true;
        return uni(ld_acquire(&reinterpret_cast<SplitSlot *>(slot_of(c))->left)) == kWarps;
    };

    uint32_t n_swept = 0, n_passed = 0, n_all = 0;  // counters of this warp
    if (warp == 0) bring(0);
    for (uint32_t chunk = 0; wait_for(&ctl.ready, chunk + 1);) {
        unsigned char *base = slot_of(chunk);
        SplitSlot &sl = *reinterpret_cast<SplitSlot *>(base);
        if (uni(sl.end)) break;
        uint32_t idx = 0;
        if (lane == 0) idx = atomicAdd(&sl.next, 1u);
        idx = uni(idx);
        if (idx >= uni(sl.n_tiles)) {
            __syncwarp();
            if (lane == 0) red_release(&sl.left, 1u);
            __syncwarp();
            chunk++;
            continue;
        }
        bool owe = idx == sl.n_tiles - 1;  // this warp brings the next chunk
        if (owe && slot_free(chunk + 1)) {
            bring(chunk + 1);
            owe = false;
        }
        const QueueDem &D = sl.dem;
        const Step<kPrec> *s_t = reinterpret_cast<const Step<kPrec> *>(base + L::table());
        const SegBound *s_seg = reinterpret_cast<const SegBound *>(base + L::seg(cap));
        const uint32_t tile = uni(sl.tile0) + idx;
        const uint32_t group = uni(sl.group), dir = group & 1u;

        if (uni((uint32_t)(sl.status == TVS_OK))) {
            const uint32_t n = uni(sl.n), n_fast = uni(sl.n_fast);
            // tiles run down stripes of 8 tile rows, so that a chunk is a compact
            // block of the DEM
            const uint32_t per = 8 * D.tiles_x, stripe = tile / per, in = tile - stripe * per;
            const uint32_t rows = min(8u, D.tiles_y - 8 * stripe);
            const uint32_t bx = in / rows, by = 8 * stripe + in - bx * rows;
            // chain k: column tx + LX (k % KX), row ty + RS (k / KX)
            const uint32_t lx = lane % LX, ly = lane / LX;
            const uint32_t tx = bx * (KX * LX) + lx;
            const uint32_t ty = D.row_begin + by * (LY * KY) + ly * LS;
            // rows past the grid are clamped, columns past it read the padding
            // after the elevations; both are discarded (and record no rings)
            auto row_ptr = [&](int r) -> const float * {
                return D.elev + (int64_t)(min(ty + RS * r, D.row_end - 1) + D.los) * D.width + tx + D.los;
            };
            uint32_t active = 0;  // chains on the grid
#pragma unroll
            for (int k = 0; k < K; k++)
                if (tx + LX * (k % KX) < D.tvs_width && ty + RS * (k / KX) < D.row_end) active |= 1u << k;
            // kernel.rs:134, the f32 observer elevation (MIXED64, FP64: the point of
            // view's own elevation; the observer height is in the step's offset)
            float hp[K];
#pragma unroll
            for (int k = 0; k < K; k++) {
                const float h = __ldg(row_ptr(k / KX) + LX * (k % KX));
                hp[k] = kWide ? h : __fadd_rn(h, D.observer_height);
            }
            f32x2 nhp[K / 2];  // negated, for the packed subtraction
#pragma unroll
            for (int q = 0; q < K / 2; q++) nhp[q] = pk(-hp[2 * q], -hp[2 * q + 1]);
            S out[K];

            // the sweep of this tile; PLAIN: a quad-layout sector that reads the
            // plain DEM (a separate instantiation, so that the quad loop is as
            // lean as without it)
            auto pass = [&](auto PLAIN) {
                constexpr bool quad = kQuad && !decltype(PLAIN)::value;
                // plain: the rows of the lane's chains (recomputed in the quad
                // layout's few plain sectors)
                const float *ep[kQuad ? 1 : KY] = {};
                if constexpr (!quad) {
#pragma unroll
                    for (int r = 0; r < (kQuad ? 1 : KY); r++) ep[r] = row_ptr(r);
                }
                // quad: the copies' base and the lane's offset in them, in bytes (rows
                // past the grid are not clamped: the copies hold zero rows for
                // them).  The copies lie within 2^31 bytes (quad_fits): a sample's
                // address is a uniform base and one 32-bit add.
                const char *qbase = nullptr;
                uint32_t qlane = 0;
                if constexpr (quad) {
                    const uint64_t q = reinterpret_cast<uint64_t>(D.quad);
                    qbase = reinterpret_cast<const char *>((uint64_t)uni((uint32_t)(q >> 32)) << 32 |
                                                           uni((uint32_t)q));
                    qlane = (((ty + D.los - ((D.row_begin + D.los) & 3u)) / 4) * D.width + tx + D.los) * 16u;
                }
                (void)qbase;
                (void)qlane;
                auto at = [&](int off, int k) -> const float * {
                    const float *row = kQuad ? row_ptr(k / KX) : ep[k / KX];
                    return row + off + LX * (k % KX);
                };
                auto quad_at = [&](int off) -> const float4 * {
                    return reinterpret_cast<const float4 *>(qbase + (qlane + (uint32_t)off));
                };
                // the four chains' samples at a step's offset
                auto load = [&](int off, float (&h)[K]) {
                    if constexpr (quad) {
                        const float4 v = __ldg(quad_at(off));
                        h[0] = v.x;
                        h[1] = v.y;
                        h[2] = v.z;
                        h[3] = v.w;
                    } else {
#pragma unroll
                        for (int k = 0; k < K; k++) h[k] = __ldg(at(off, k));
                    }
                };
                auto load1 = [&](int off, int k) -> float {
                    if constexpr (quad) return __ldg(reinterpret_cast<const float *>(quad_at(off)) + k);
                    else return __ldg(at(off, k));
                };
                // ring records: the step's offset in the DEM, chain k's kernel id, and
                // the DEM id of its sample (ids fit an int); a call over several
                // sectors keeps each sector's records apart: its sector s owns records
                // s * total_bands ..
                auto orig = [&](uint32_t st) -> int {
                    if constexpr (kPrec == TVS_PRECISION_EXACT32 || kMix) {
                        return s_t[st + kAhead].orig;
                    } else if constexpr (quad) {
                        const int o =
                            __ldg(&D.offs[(uint64_t)(a.first_sector + (group >> 1)) * D.step_cap + st].x);
                        return dir ? -o : o;
                    } else {
                        return s_t[st].next;
                    }
                };
                auto kid = [&](int k) -> uint64_t {
                    return (uint64_t)(ty + RS * (k / KX)) * D.tvs_width + tx + LX * (k % KX) +
                           (dir ? a.half_bands : 0) +
                           (uint64_t)(a.first_sector - a.first_record_sector + (group >> 1)) * 2 * a.half_bands;
                };
                // the lane's first record, and chain k's from it (one 32-bit add and a
                // wide multiply-add per id in place of two 64-bit products)
                uint32_t *ring0 = nullptr;
                uint32_t pov0 = 0, row_ids = 0, row_slots = 0, col_slots = 0;
                if constexpr (kRings) {
                    ring0 = a.rings + kid(0) * a.ring_reserved;
                    pov0 = (ty + D.los) * D.width + tx + D.los;
                    row_ids = RS * D.width;
                    row_slots = RS * D.tvs_width * a.ring_reserved;
                    col_slots = LX * a.ring_reserved;
                }
                auto dem_id = [&](int k, int o) -> uint32_t {
                    return pov0 + (uint32_t)(k / KX) * row_ids + LX * (k % KX) + (uint32_t)o;
                };
                auto ring_put = [&](int k, uint32_t slot, uint32_t value) {
                    if (slot < a.ring_reserved) {
                        ring0[(k / KX) * row_slots + (k % KX) * col_slots + slot] = value;
                    } else {
                        const uint64_t band = kid(k);
                        const uint32_t at_ = atomicAdd(&a.ring_counters[0], 1u);
                        if (at_ < a.spill_cap)
                            a.spill[at_] = make_uint4((uint32_t)band, (uint32_t)(band >> 32), slot, value);
                    }
                };
                uint32_t nr[K];        // ring ids so far (kernel.rs:113 starts at 1)
                uint32_t prev = 0xFu;  // visibility at the previous step (kernel.rs:146)
                if constexpr (kRings) {
#pragma unroll
                    for (int k = 0; k < K; k++) {
                        nr[k] = 1;
                        if (active >> k & 1u) ring_put(k, 1, dem_id(k, 0));  // kernel.rs:145
                    }
                } else {
                    prev = 0;
                }
                auto events = [&](uint32_t vis, uint32_t st) {
                    const uint32_t ev = (vis ^ prev) & active;
                    if (__any_sync(0xffffffffu, ev != 0)) {
                        const int o = orig(st);
#pragma unroll
                        for (int k = 0; k < K; k++)
                            if (ev >> k & 1u) ring_put(k, ++nr[k], dem_id(k, o));
                        __syncwarp();
                    }
                    prev = vis;
                };
                // no chain is visible at step st
                auto close = [&](uint32_t st) {
                    if constexpr (kRings) events(0, st);
                };
                // The largest elevation any lane of this warp samples in a
                // segment: the block maxima over the warp's patch of points of
                // view moved by the segment's offset range (warp-uniform).
                auto segment_max = [&](const SegBound &b) -> float {
                    const int px0 = (int)(bx * (KX * LX) + D.los), px1 = px0 + KX * LX - 1;
                    const int py0 = (int)(D.row_begin + by * (LY * KY) + D.los), py1 = py0 + LY * KY - 1;
                    const int bx0 = max(px0 + b.x0, 0) / (int)kBlockMax;
                    const int bx1 = min(max(px1 + b.x1, 0) / (int)kBlockMax, (int)D.bmax_w - 1);
                    const int by0 = max(py0 + b.y0, 0) / (int)kBlockMax;
                    const int by1 = min(max(py1 + b.y1, 0) / (int)kBlockMax, (int)D.bmax_h - 1);
                    float m = -INFINITY;
                    // 8 x 4 blocks at a time
                    for (int y0 = by0; y0 <= by1; y0 += 4)
                        for (int x0 = bx0; x0 <= bx1; x0 += 8) {
                            const int y = y0 + (int)(lane >> 3), x = x0 + (int)(lane & 7u);
                            if (y <= by1 && x <= bx1)
                                m = fmaxf(m, __ldg(D.bmax + (uint32_t)y * D.bmax_w + x));
                        }
                    return warp_max(m);
                };
                // A segment can be skipped when no chain can change state at
                // any of its steps (in a wide sector never): every sample h <= B, so e <= RN(B - h_pov)
                // and the first test's value fma(e, y, z) is at most
                // fma(RN(B - h_pov), y_max or y_min, z_max) (RN and fma are
                // monotone).  A chain visible at the previous step closes its ring
                // at the segment's first one.
                auto skippable = [&](uint32_t seg, auto &&below) -> bool {
                    const SegBound b = s_seg[seg];
                    const float B = segment_max(b);
                    bool skip = true;
#pragma unroll
                    for (int k = 0; k < K; k++) {
                        const float E = __fsub_rn(B, hp[k]);
                        skip &= below(k, __fmaf_rn(E, E >= 0.0f ? b.ymax : b.ymin, b.zmax));
                    }
                    return __all_sync(0xffffffffu, skip);
                };
                // e = h - h_pov and the estimate fma(e, y, z) of the four chains (the
                // subtraction packed; the multiply-adds not, for they would need
                // y and z in pairs)
                auto estimate = [&](const float (&h)[K], float y, float z, float (&e)[K], float (&f)[K]) {
#pragma unroll
                    for (int q = 0; q < K / 2; q++)
                        upk(add2(pk(h[2 * q], h[2 * q + 1]), nhp[q]), e[2 * q], e[2 * q + 1]);
#pragma unroll
                    for (int k = 0; k < K; k++) f[k] = __fmaf_rn(e[k], y, z);
                };
                uint32_t i = 0;
                // The segments of fast steps, two steps an iteration: the samples of
                // step i + 2 take the registers of step i's as soon as its estimates
                // are formed, so two loads are under way at every step (one step
                // ahead: 1201^2 exact f32 4.47 ms, two: 3.74 ms).
                auto sweep_fast = [&](auto &&below, auto &&step) {
                    for (uint32_t seg = 0; i < n_fast; seg++) {
                        const uint32_t i1 = min(i + kSegSteps, n_fast);
                        if (skippable(seg, below)) {
                            close(i);
                            i = i1;
                            continue;
                        }
                        n_swept += i1 - i;
                        const Step<kPrec> *p = s_t + i + kAhead;
                        float h0[K];
                        load(s_t[i].next, h0);
                        if constexpr (kRings) {
#pragma unroll 1
                            for (; i < i1; i++, p++) step(i, p, h0);
                            continue;
                        }
                        float h1[K];
                        load(s_t[i + 1].next, h1);
                        // four an iteration where the registers allow it (1201^2 exact f32
                        // 3.66 -> 3.56 ms, 3601^2 FP32 64.1 -> 61.8; MIXED64 spills)
                        if constexpr (!kWide) {
                            for (; i + 4 <= i1; i += 4, p += 4) {
                                step(i, p, h0);
                                step(i + 1, p + 1, h1);
                                step(i + 2, p + 2, h0);
                                step(i + 3, p + 3, h1);
                            }
                        }
#pragma unroll 1
                        for (; i + 2 <= i1; i += 2, p += 2) {
                            step(i, p, h0);
                            step(i + 1, p + 1, h1);
                        }
                        if (i < i1) {
                            step(i, p, h0);
                            i++;
                        }
                    }
                };
                if constexpr (kFp32) {
                    // ---- the reciprocal-table form: the estimate is the angle --
                    float m[K], sf[K];
#pragma unroll
                    for (int k = 0; k < K; k++) {
                        m[k] = active >> k & 1u ? kMaxAngle : INFINITY;  // off the grid: never visible
                        sf[k] = 0.0f;
                    }
                    // step i from its samples h, which then hold step i + kAhead's
                    auto step = [&](uint32_t st, const Step<kPrec> *p, float (&h)[K]) {
                        const Step<kPrec> t = *p;
                        float e[K], ang[K];
                        estimate(h, t.y, t.z, e, ang);
                        load(t.next, h);
                        [[maybe_unused]] uint32_t vis = 0;
#pragma unroll
                        for (int k = 0; k < K; k++) {
                            if constexpr (kRings) vis |= (uint32_t)(ang[k] > m[k]) << k;
                            raise_fp32(ang[k], m[k], sf[k], t.w);
                        }
                        if constexpr (kRings) events(vis, st);
                    };
                    sweep_fast([&](int k, float bound) { return bound <= m[k]; }, step);
                    for (; i < n; i++) {  // zero distances: y = inf, the same form
                        float h[K];
                        load(s_t[i].next, h);
                        step(i, s_t + i + kAhead, h);
                    }
#pragma unroll
                    for (int k = 0; k < K; k++) out[k] = sf[k];
                } else if constexpr (kF64) {
                    // ---- FP64: angles in double where the first test passes -----
                    // its threshold lo = RN(m) - 2^-20 |RN(m)| leaves 2.6 x the
                    // estimate's error relative to the angle, as the guard band does
                    double m[K], acc[K];
                    float lo[K];
#pragma unroll
                    for (int k = 0; k < K; k++) {
                        // off the grid: above every angle, and finite (an infinite m makes lo
                        // a NaN at the warp's first passing step, below which no bound
                        // lies: the tile then skipped no segment any more)
                        const float first = active >> k & 1u ? kMaxAngle : FLT_MAX;
                        m[k] = (double)first;
                        lo[k] = __fmaf_rn(fabsf(first), -kRel, first);
                        acc[k] = 0.0;
                    }
                    const double o64 = (double)D.observer_height;
                    auto step = [&](uint32_t st, const Step<kPrec> *p, float (&h)[K]) {
                        const float y = p->y, z = p->z;
                        const int next = p->next;
                        float e[K], f[K], hs[K];
                        estimate(h, y, z, e, f);
#pragma unroll
                        for (int k = 0; k < K; k++) hs[k] = h[k];
                        load(next, h);
                        bool hit = false;
#pragma unroll
                        for (int k = 0; k < K; k++) hit |= f[k] >= lo[k];
                        if (__any_sync(0xffffffffu, hit)) {
                            n_passed++;
                            const double d = (double)p->d, y64 = p->y64, c64 = p->c64;
                            const double w = __dmul_rn(d, 0.0174533);  // kernel.rs:216
                            // (every chain: a vote per chain to leave out the ones below
                            // the test measured 6.71 against 6.30 ms at 1201^2)
#pragma unroll
                            for (int k = 0; k < K; k++) {
                                const double hp64 = __dadd_rn((double)hp[k], o64);
                                const double ang = __dsub_rn(
                                    div_table64(__dsub_rn((double)hs[k], hp64), y64, d), c64);
                                const bool v = ang > m[k];  // false for a NaN: m stays (f64::max)
                                acc[k] = __fma_rn(w, __hiloint2double(v ? 0x3ff00000 : 0, 0), acc[k]);
                                m[k] = v ? ang : m[k];
                                const float m32 = __double2float_rn(m[k]);
                                lo[k] = __fmaf_rn(fabsf(m32), -kRel, m32);
                            }
                        }
                    };
                    sweep_fast([&](int k, float bound) { return bound < lo[k]; }, step);
                    for (; i < n; i++) {  // past the table division's domain: IEEE division
                        const double4 *q = D.dtab + (uint64_t)(a.first_sector + (group >> 1)) * D.step_cap + i;
                        const double c64 = __ldg(&q->y), w = __ldg(&q->z), d = __ldg(&q->w);
                        float h[K];
                        load(s_t[i].next, h);
#pragma unroll
                        for (int k = 0; k < K; k++) {
                            const double hp64 = __dadd_rn((double)hp[k], o64);
                            const double ang = __dsub_rn(__ddiv_rn(__dsub_rn((double)h[k], hp64), d), c64);
                            if (ang > m[k]) acc[k] = __dadd_rn(acc[k], w);
                            m[k] = fmax(ang, m[k]);
                        }
                    }
#pragma unroll
                    for (int k = 0; k < K; k++) out[k] = acc[k];
                } else if constexpr (!kMix) {
                    // ---- exact f32, the running maximum held exactly ----------
                    // where the first test passes the reference's angle is computed
                    // for every chain (kernel.rs:175-233)
                    float m[K], lo[K], sf[K];
#pragma unroll
                    for (int k = 0; k < K; k++) {
                        m[k] = active >> k & 1u ? kMaxAngle : INFINITY;  // off the grid: never visible
                        lo[k] = active >> k & 1u ? __fmaf_rn(fabsf(m[k]), -kRelExact, m[k]) : INFINITY;
                        sf[k] = 0.0f;
                    }
                    auto step = [&](uint32_t st, const Step<kPrec> *p, float (&h)[K]) {
                        const float y = p->y, z = p->z, w = p->w;
                        const int next = p->next;
                        float e[K], f[K];
                        estimate(h, y, z, e, f);  // kernel.rs:164
                        load(next, h);
                        bool hit = false;
#pragma unroll
                        for (int k = 0; k < K; k++) hit |= f[k] >= lo[k];
                        if (__any_sync(0xffffffffu, hit)) {
                            n_passed++;
                            const float d = p->d, c = p->c;
                            [[maybe_unused]] uint32_t vis = 0;
#pragma unroll
                            for (int k = 0; k < K; k++) {
                                const float ang = __fsub_rn(div_table32(e[k], y, d), c);
                                if constexpr (kRings) vis |= (uint32_t)(ang > m[k]) << k;
                                raise_exact(ang, m[k], sf[k], lo[k], w);
                            }
                            if constexpr (kRings) events(vis, st);
                        } else {
                            close(st);
                        }
                    };
                    sweep_fast([&](int k, float bound) { return bound < lo[k]; }, step);
                    for (; i < n; i++) {  // past the table division's domain: IEEE division
                        const Step<kPrec> &t = s_t[i + kAhead];
                        const bool fast = t.d >= 0x1p-20f && t.d <= 0x1p20f;
                        float h[K];
                        load(s_t[i].next, h);
                        uint32_t vis = 0;
#pragma unroll
                        for (int k = 0; k < K; k++) {
                            const float e = __fsub_rn(h[k], hp[k]);
                            const float ang =
                                __fsub_rn(fast ? div_table32(e, t.y, t.d) : __fdiv_rn(e, t.d), t.c);
                            const bool v = ang > m[k];
                            if (v) {
                                sf[k] = __fadd_rn(sf[k], t.w);
                                m[k] = ang;
                            }
                            vis |= (uint32_t)v << k;
                        }
                        if constexpr (kRings) events(vis, i);
                    }
#pragma unroll
                    for (int k = 0; k < K; k++) out[k] = sf[k];
                } else {
                    // ---- MIXED64: the guard band ------------------------------
                    float nmid[K], hw[K];  // -(the maximum's estimate), the band's half width
                    // step of the running maximum, 16 bits, two chains per register
                    // (0xffff: the initial maximum)
                    uint32_t jpk[K / 2];
                    double acc[K];
                    const float first = s_t[kAhead].band;
#pragma unroll
                    for (int k = 0; k < K; k++) {
                        // the initial maximum is -2000; chains off the grid are never
                        // visible
                        nmid[k] = active >> k & 1u ? -kMaxAngle : -INFINITY;
                        hw[k] = active >> k & 1u ? __fmaf_rn(2000.0f, kRel, first) : 0.0f;
                        jpk[k / 2] = 0xffffffffu;
                        acc[k] = 0.0;
                    }
                    auto getj = [&](int k) -> int32_t {
                        const uint32_t v = (jpk[k / 2] >> (16 * (k & 1))) & 0xffffu;
                        return v == 0xffffu ? -1 : (int32_t)v;
                    };
                    const double4 *gdt = D.dtab + (uint64_t)(a.first_sector + (group >> 1)) * D.step_cap;
                    auto step = [&](uint32_t st, const Step<kPrec> *p, float (&h)[K]) {
                        const float y = p->y, z = p->z, band = p->band;
                        const int next = p->next;
                        float e[K], f[K], x[K];
                        estimate(h, y, z, e, f);
                        load(next, h);
#pragma unroll
                        for (int q = 0; q < K / 2; q++)
                            upk(add2(pk(f[2 * q], f[2 * q + 1]), pk(nmid[2 * q], nmid[2 * q + 1])),
                                x[2 * q], x[2 * q + 1]);
                        bool hit = false;
#pragma unroll
                        for (int k = 0; k < K; k++) hit |= x[k] >= -hw[k];
                        if (__any_sync(0xffffffffu, hit)) {
                            n_passed++;
                            const double w = p->w;
                            bool amb = false;  // inside the band
#pragma unroll
                            for (int k = 0; k < K; k++) amb |= fabsf(x[k]) <= hw[k];
                            [[maybe_unused]] uint32_t vis = 0;
                            if (__any_sync(0xffffffffu, amb)) {
                                uint32_t n_amb = 0;
#pragma unroll
                                for (int k = 0; k < K; k++) {
                                    if (!(x[k] >= -hw[k])) continue;
                                    if (fabsf(x[k]) <= hw[k]) {
                                        n_amb++;
                                        const int32_t j = getj(k);
                                        if (!mix_visible(load1(s_t[st].next, k), load1(s_t[max(j, 0)].next, k),
                                                         hp[k], D.observer_height, gdt, st, j))
                                            continue;
                                    }
                                    nmid[k] = -f[k];
                                    hw[k] = __fmaf_rn(fabsf(f[k]), kRel, band);
                                    jpk[k / 2] = __byte_perm(jpk[k / 2], st, (k & 1) ? 0x5410 : 0x3254);
                                    acc[k] = __dadd_rn(acc[k], w);
                                    vis |= 1u << k;
                                }
                                if (n_amb) atomicAdd(&ctl.diag[3], (unsigned long long)n_amb);
                                __syncwarp();
                            } else {
                                // outside the band the larger estimate is the maximum's
                                if constexpr (kRings) {
#pragma unroll
                                    for (int k = 0; k < K; k++) vis |= (uint32_t)(x[k] >= -hw[k]) << k;
                                }
                                raise_mix<0>(x[0], f[0], band, st, w, hw[0], jpk[0], acc[0]);
                                raise_mix<1>(x[1], f[1], band, st, w, hw[1], jpk[0], acc[1]);
                                raise_mix<0>(x[2], f[2], band, st, w, hw[2], jpk[1], acc[2]);
                                raise_mix<1>(x[3], f[3], band, st, w, hw[3], jpk[1], acc[3]);
#pragma unroll
                                for (int k = 0; k < K; k++) nmid[k] = fminf(nmid[k], -f[k]);  // a NaN leaves it
                            }
                            if constexpr (kRings) events(vis, st);
                        } else {
                            close(st);
                        }
                    };
                    sweep_fast([&](int k, float bound) { return __fadd_rn(bound, nmid[k]) < -hw[k]; }, step);
                    // the steps past the table-division domain (the zero
                    // distances): exact arithmetic from the exact maximum
                    if (i < n) {
                        double m[K];
#pragma unroll
                        for (int k = 0; k < K; k++) {
                            const int32_t j = getj(k);
                            m[k] = kMaxAngle;
                            if (j >= 0)
                                m[k] = mix_angle(load1(s_t[j].next, k), hp[k], D.observer_height, gdt,
                                                 (uint32_t)j);
                        }
                        __syncwarp();
                        for (; i < n; i++) {
                            const double4 q = gdt[i];
                            float hk[K];
                            load(s_t[i].next, hk);
                            uint32_t vis = 0;
#pragma unroll
                            for (int k = 0; k < K; k++) {
                                const double hp64 = __dadd_rn((double)hp[k], (double)D.observer_height);
                                const double ang =
                                    __dsub_rn(__ddiv_rn(__dsub_rn((double)hk[k], hp64), q.w), q.y);
                                const bool v = ang > m[k];
                                if (v) acc[k] = __dadd_rn(acc[k], q.z);
                                m[k] = fmax(ang, m[k]);
                                vis |= (uint32_t)v << k;
                            }
                            if constexpr (kRings) events(vis, i);
                        }
                    }
#pragma unroll
                    for (int k = 0; k < K; k++) out[k] = acc[k];
                }
                if constexpr (kRings) {
                    // kernel.rs:237-243: close a ring cut off by the line of
                    // sight, then the count in slot 0
                    const int o_last = n ? orig(n - 1) : 0;
                    uint32_t most = 0, over = 0;
#pragma unroll
                    for (int k = 0; k < K; k++) {
                        if (!(active >> k & 1u)) continue;
                        if (prev >> k & 1u) ring_put(k, ++nr[k], dem_id(k, o_last));
                        if (a.ring_lens) a.ring_lens[kid(k)] = nr[k];
                        else ring_put(k, 0, nr[k]);
                        most = max(most, nr[k]);
                        over += nr[k] >= a.ref_reserved;
                    }
                    most = __reduce_max_sync(0xffffffffu, most);
                    over = __reduce_add_sync(0xffffffffu, over);
                    if (lane == 0) {
                        if (over) atomicAdd(&a.ring_counters[1], over);
                        if (most) atomicMax(&a.ring_counters[2], most);
                    }
                }
            };
            if constexpr (kQuad) {
                if (uni(sl.plain)) pass(std::true_type{});
                else pass(std::false_type{});
            } else {
                pass(std::false_type{});
            }
            n_all += n_fast;

            // ---- the surfaces, in order ---------------------------------------
            auto point = [&](int k) -> uint64_t {
                return (uint64_t)(ty + RS * (k / KX)) * D.tvs_width + tx + LX * (k % KX);
            };
            if (a.planes) {
                S *plane = reinterpret_cast<S *>(a.planes) +
                           ((size_t)group * a.tiles_per_sector + D.done_base + tile) * (32 * K) + lane;
#pragma unroll
                for (int k = 0; k < K; k++) __stcg(plane + 32 * k, out[k]);
            } else {
                // the tile's previous item must be complete
                bool ok = true;
                if (group > 0) {
                    const volatile uint32_t *d = a.done + D.done_base + tile;
                    const volatile int32_t *err = a.error;
                    uint32_t spins = 0;
                    while (!__all_sync(0xffffffffu, *d >= group)) {
                        // give up at the limit, or soon when another wait already did
                        spins++;
                        if (spins > a.spin_limit ||
                            ((spins & 15u) == 0 && __any_sync(0xffffffffu, *err != 0))) {
                            if (lane == 0) atomicExch(a.error, (int32_t)TVS_ERR_TIMEOUT);
                            ok = false;
                            break;
                        }
                        __nanosleep(256);
                    }
                    __threadfence();
                    __syncwarp();
                }
#pragma unroll
                for (int k = 0; k < K; k++) {
                    if (!ok || !(active >> k & 1u)) continue;
                    const uint64_t p = point(k);
                    // in L2: another SM wrote the previous item's values
                    if constexpr (kWide) {
                        const double cum = __dadd_rn(__ldcg(D.cumulative64 + p), out[k]);
                        __stcg(D.cumulative64 + p, cum);
                        if (dir) {
                            const float c32 = __double2float_rn(cum);
                            __stcg(D.cumulative + p, c32);
                            if (D.total) __stcg(D.total + p, __fadd_rn(__ldcg(D.total + p), c32));
                        }
                    } else {
                        const float cum = __fadd_rn(__ldcg(D.cumulative + p), out[k]);
                        __stcg(D.cumulative + p, cum);
                        if (dir && D.total)  // compute.rs:206-214
                            __stcg(D.total + p, __fadd_rn(__ldcg(D.total + p), cum));
                    }
                }
            }
        }
        if (!a.planes) {
            __threadfence();  // this lane's surface writes before the tile's counter
            __syncwarp();
            if (lane == 0 && D.done_base + tile != a.held_tile)
                atomicAdd(a.done + D.done_base + tile, 1u);
        } else {
            // Release only: an acquiring fence invalidates the SM's L1, which holds
            // the DEM for 32 warps; one per tile and launch (the last item's below)
            // does, one per item left 37-48 % of the sectors hitting.
            __syncwarp();
            uint32_t before = 0;
            if (lane == 0) before = add_release(a.done + D.done_base + tile, 1u);
            before = uni(before);
            if (before == 2 * a.n_sectors - 1) {
                // the tile's last item: its planes of every sector, in order
                __threadfence();
                __syncwarp();
                const uint32_t per = 8 * D.tiles_x, stripe = tile / per, in = tile - stripe * per;
                const uint32_t rows = min(8u, D.tiles_y - 8 * stripe);
                const uint32_t bx = in / rows, by = 8 * stripe + in - bx * rows;
                const uint32_t tx = bx * (KX * LX) + lane % LX;
                const uint32_t ty = D.row_begin + by * (LY * KY) + lane / LX * LS;
                const size_t stride = (size_t)a.tiles_per_sector * (32 * K);  // between groups
                const S *plane = reinterpret_cast<const S *>(a.planes) +
                                 (size_t)(D.done_base + tile) * (32 * K) + lane;
                bool on[K];
                uint64_t p[K];
                S cum[K];
                float total[K], c32[K];
#pragma unroll
                for (int k = 0; k < K; k++) {
                    const uint32_t col = tx + LX * (k % KX), row = ty + RS * (k / KX);
                    on[k] = col < D.tvs_width && row < D.row_end;
                    p[k] = on[k] ? (uint64_t)row * D.tvs_width + col : 0;
                    if constexpr (kWide) cum[k] = on[k] ? __ldcg(D.cumulative64 + p[k]) : 0.0;
                    else cum[k] = on[k] ? __ldcg(D.cumulative + p[k]) : 0.0f;
                    total[k] = on[k] && D.total ? __ldcg(D.total + p[k]) : 0.0f;
                    c32[k] = 0.0f;
                }
                bool any = false;
                constexpr int kAhead = 2;  // sectors whose planes are read together
                for (uint32_t s0 = 0; s0 < a.n_sectors; s0 += kAhead) {
                    S f[kAhead][K], b[kAhead][K];
                    bool ok[kAhead];
#pragma unroll
                    for (int q = 0; q < kAhead; q++) {
                        const uint32_t s = s0 + q;
                        ok[q] = s < a.n_sectors && __ldg(&D.hdr[a.first_sector + s].status) == TVS_OK;
#pragma unroll
                        for (int k = 0; k < K; k++) {
                            f[q][k] = ok[q] ? __ldcg(plane + (size_t)(2 * s) * stride + 32 * k) : (S)0;
                            b[q][k] = ok[q] ? __ldcg(plane + (size_t)(2 * s + 1) * stride + 32 * k) : (S)0;
                        }
                    }
#pragma unroll
                    for (int q = 0; q < kAhead; q++) {
                        if (!ok[q]) continue;
                        any = true;
#pragma unroll
                        for (int k = 0; k < K; k++) {
                            if constexpr (kWide) {
                                cum[k] = __dadd_rn(__dadd_rn(cum[k], f[q][k]), b[q][k]);
                                c32[k] = __double2float_rn(cum[k]);
                            } else {
                                cum[k] = __fadd_rn(__fadd_rn(cum[k], f[q][k]), b[q][k]);
                                c32[k] = cum[k];
                            }
                            total[k] = __fadd_rn(total[k], c32[k]);  // compute.rs:206-214
                        }
                    }
                }
#pragma unroll
                for (int k = 0; k < K; k++) {
                    if (!on[k] || !any) continue;
                    if constexpr (kWide) __stcg(D.cumulative64 + p[k], cum[k]);
                    __stcg(D.cumulative + p[k], c32[k]);
                    if (D.total) __stcg(D.total + p[k], total[k]);
                }
            }
        }
        if (owe) {  // the next chunk's slot was still in use
            bool ok = true;
            if (chunk + 1 >= n_slots)
                ok = wait_for(&reinterpret_cast<SplitSlot *>(slot_of(chunk + 1))->left, kWarps);
            if (!ok) break;
            bring(chunk + 1);
        }
    }
    if (a.diag && lane == 0) {
        atomicAdd(&ctl.diag[0], (unsigned long long)n_swept);
        atomicAdd(&ctl.diag[1], (unsigned long long)n_passed);
        atomicAdd(&ctl.diag[2], (unsigned long long)n_all);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (a.diag)
            for (int q = 0; q < 3; q++) atomicAdd(&a.diag[q], ctl.diag[q]);
        if (a.rechecks && ctl.diag[3]) atomicAdd(a.rechecks, ctl.diag[3]);
    }
}

// Chunks in the ring: three where they leave the SM's CTAs room, else two.
template <int kPrec, bool kRings>
cudaError_t ring_slots(uint32_t step_cap, uint32_t *n_slots) {
    int dev = 0, per_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess)
        e = cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    const size_t three = SplitSmem<kPrec>::total(step_cap, 3) * split_min_blocks<kPrec, kRings>();
    *n_slots = three <= (size_t)per_sm / 2 ? 3 : 2;
    return e;
}

template <int kPrec, int kLayout, bool kRings>
cudaError_t launch_split_t(const QueueArgs &a, cudaStream_t s) {
    uint32_t n_slots = 2;
    const cudaError_t e = ring_slots<kPrec, kRings>(a.max_step_cap, &n_slots);
    if (e != cudaSuccess) return e;
    const size_t smem = SplitSmem<kPrec>::total(a.max_step_cap, n_slots);
    return launch_persistent(
        reinterpret_cast<const void *>(&k_sweep_split<kPrec, kLayout, kRings>), a,
        (uint64_t)a.chunks * a.n_sectors * 2, dim3(32 * split_warps<kPrec, kRings>()), smem, s, n_slots);
}

template <int kPrec, bool kRings>
cudaError_t launch_split_layout(const QueueArgs &a, int layout, cudaStream_t s) {
    switch (layout) {
    case 1: return launch_split_t<kPrec, 1, kRings>(a, s);
    case 2: return launch_split_t<kPrec, 2, kRings>(a, s);
    case 3: return launch_split_t<kPrec, 3, kRings>(a, s);
    case 4: return launch_split_t<kPrec, 4, kRings>(a, s);
    case 5: return launch_split_t<kPrec, 5, kRings>(a, s);
    case 6: return launch_split_t<kPrec, 6, kRings>(a, s);
    case 7: return launch_split_t<kPrec, 7, kRings>(a, s);
    case 8: return launch_split_t<kPrec, 8, kRings>(a, s);
    case 9: return launch_split_t<kPrec, 9, kRings>(a, s);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace

cudaError_t launch_persistent(const void *fn, const QueueArgs &a, uint64_t items, dim3 block,
                              size_t smem, cudaStream_t s, uint32_t n_slots) {
    struct Occ {
        size_t attr = 0, smem = 0;
        int blocks = -1;
    };
    static std::mutex mu;
    static std::map<std::pair<const void *, int>, Occ> occ;
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    int blocks_per_sm;
    {
        // contexts on several devices or host threads may launch this kernel
        // concurrently: the attribute only grows, so a launch never finds it
        // below its own shared memory
        std::lock_guard<std::mutex> lock(mu);
        Occ &o = occ[std::make_pair(fn, dev)];
        if (smem > o.attr) {
            e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (e != cudaSuccess) return e;
            o.attr = smem;
        }
        if (o.blocks < 0 || o.smem != smem) {
            // The resident CTAs at the largest shared-memory carveout, then the
            // smallest carveout that still holds them: the rest of the SM's
            // 256 KB stays L1 cache for the DEM samples (left to itself the
            // driver sizes the carveout for more CTAs than the registers allow).
            int b = 0, per_sm = 0, reserved = 0;
            e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
            if (e == cudaSuccess)
                e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, fn, (int)(block.x * block.y), smem);
            if (e == cudaSuccess)
                e = cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
            if (e == cudaSuccess)
                e = cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev);
            if (e != cudaSuccess) return e;
            b = b < 1 ? 1 : b;
            if (per_sm > 0) {
                const size_t need = (size_t)b * (smem + (size_t)reserved);
                const int pct = (int)std::min<size_t>(100, (need * 100 + per_sm - 1) / per_sm);
                int b2 = 0;
                e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, pct);
                if (e == cudaSuccess)
                    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b2, fn, (int)(block.x * block.y), smem);
                if (e != cudaSuccess) return e;
                if (b2 < b) {  // the rounding lost a CTA: keep the largest carveout
                    e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
                    if (e != cudaSuccess) return e;
                }
            }
            o.blocks = b;
            o.smem = smem;
        }
        blocks_per_sm = o.blocks;
    }
    if (a.done_total > a.done_cap || a.done != a.queue + 1) return cudaErrorInvalidValue;
    // the tile counters follow the queue counter in memory
    e = cudaMemsetAsync(a.queue, 0, ((size_t)a.done_total + 1) * sizeof(uint32_t), s);
    if (e != cudaSuccess) return e;
    const uint32_t grid = (uint32_t)std::min<uint64_t>((uint64_t)blocks_per_sm * sms, items);
    QueueArgs args = a;
    void *params[] = {&args, &n_slots};  // (the row kernels take the first only)
    e = cudaLaunchKernel(fn, dim3(grid), block, params, smem, s);
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

size_t split_plane_bytes(int precision, const QueueConfig &c, uint32_t tiles_per_sector,
                         uint32_t n_sectors, uint32_t *sectors) {
    *sectors = 0;
    if (c.layout == 0 || tiles_per_sector == 0) return 0;
    const size_t one = precision == TVS_PRECISION_MIXED64 || precision == TVS_PRECISION_FP64
                           ? sizeof(double) : sizeof(float);
    const size_t sector = (size_t)2 * tiles_per_sector * 32 * K * one;
    // launches of about even size
    const size_t budget = std::min(kPlaneBytesMost, std::max(kPlaneBytes, kPlaneSectors * sector));
    const size_t fit = std::min<size_t>(n_sectors, std::max<size_t>(budget / sector, 1));
    const uint32_t launches = (uint32_t)((n_sectors + fit - 1) / fit);
    *sectors = (n_sectors + launches - 1) / launches;
    return *sectors * sector;
}

cudaError_t launch_sweep_split(const QueueArgs &a, int precision, int layout, cudaStream_t s) {
    if (a.n_dems == 0 || a.tiles_per_sector == 0 || a.n_sectors == 0) return cudaSuccess;
    const bool rings = a.rings != nullptr;
    if (rings && (!a.ring_counters || !a.spill || a.ring_reserved < 2))
        return cudaErrorInvalidValue;
    switch (precision) {
    case TVS_PRECISION_EXACT32:
        return rings ? launch_split_layout<TVS_PRECISION_EXACT32, true>(a, layout, s)
                     : launch_split_layout<TVS_PRECISION_EXACT32, false>(a, layout, s);
    case TVS_PRECISION_MIXED64:
        // 16-bit steps (0xffff marks the initial maximum): at most 65535 steps,
        // a step table of at most 65536 entries (its length rounds up to 4)
        if (a.max_step_cap > 0x10000u) return cudaErrorInvalidValue;
        return rings ? launch_split_layout<TVS_PRECISION_MIXED64, true>(a, layout, s)
                     : launch_split_layout<TVS_PRECISION_MIXED64, false>(a, layout, s);
    case TVS_PRECISION_FP64:  // the quad layout's tiling only; ring records elsewhere
        if (rings) return cudaErrorInvalidValue;
        return layout == kQuadLayout     ? launch_split_t<TVS_PRECISION_FP64, kQuadLayout, false>(a, s)
               : layout == kQuadFallback ? launch_split_t<TVS_PRECISION_FP64, kQuadFallback, false>(a, s)
                                         : cudaErrorInvalidValue;
    case TVS_PRECISION_FP32:
        return rings ? launch_split_layout<TVS_PRECISION_FP32, true>(a, layout, s)
                     : launch_split_layout<TVS_PRECISION_FP32, false>(a, layout, s);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace tvs
