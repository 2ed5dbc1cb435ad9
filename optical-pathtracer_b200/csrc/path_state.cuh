// Path state of the wavefront loop: structure-of-arrays in HBM, one slot per path in flight, and
// the queues that join the kernels.
#pragma once

#include "device_scene.cuh"
#include "rng.cuh"
#include "traverse.cuh"

namespace owec {

// Precision modes (owec.h OWEC_PRECISION_*): R is the arithmetic of directions, throughput and
// optics; Ro the analytic roots; Rr their refinement; origins are FP64 unless PlainOrigin.
template <int M> struct Mode;
template <> struct Mode<OWEC_PRECISION_MIXED> {
    using R = float; using Ro = float; using Rr = double; static constexpr bool plainOrigin = false;
};
template <> struct Mode<OWEC_PRECISION_FP32> {
    using R = float; using Ro = float; using Rr = float; static constexpr bool plainOrigin = true;
};
template <> struct Mode<OWEC_PRECISION_FP64> {
    using R = double; using Ro = double; using Rr = double; static constexpr bool plainOrigin = false;
};

// The ray a path travels next, and what the intersect kernel needs of it.
template <class R>
struct alignas(16) PathRay {
    double o[3];      // camera-relative origin (rounded to FP32 after every update in the plain mode)
    R d[3];
    uint32_t region;  // region the ray travels in
    uint32_t depB;    // boundary and primitive it left (kNone)
    uint32_t depP;
    float errN;       // its anchor's error normal to a surface
};

// Throughput and spectral state.
template <class R>
struct alignas(16) PathSpec {
    R beta[4];
    float lambda[4];
    float pdf[4];     // 0: terminated secondary
    float L[4];       // radiance gathered so far
};

// Bookkeeping of a path.
struct alignas(16) PathAux {
    uint64_t rngState;
    uint32_t stream;    // PCG32 stream (the pass index of this sample)
    uint32_t pixel;
    uint32_t depth;     // bounce count (the reference's loop variable)
    uint32_t flags;     // kFlagSpecular | kFlagAlive
    float prevPdf;
    float weight;       // detector importance / pdf
    double prevP[3];    // last scattering vertex (camera-relative FP64: emission MIS decides inside or
                        // outside an emitting sphere from it, which FP32 rounding can flip)
    uint32_t lastBoundary;
};
constexpr uint32_t kFlagSpecular = 1u, kFlagAlive = 2u;

// Path state passes through the L2 once per kernel, far more of it than the L2 holds. Its loads and
// stores are marked evict-first (ld.global.cs / st.global.cs), so that it does not displace the
// BVH nodes and primitives, which every traversal kernel reads again.
#ifndef OWEC_STREAM_STATE
#define OWEC_STREAM_STATE 1
#endif
template <class T>
__device__ __forceinline__ T loadStream(const T* p) {
#if OWEC_STREAM_STATE
    if constexpr (alignof(T) >= 16 && sizeof(T) % 16 == 0) {
        constexpr int n = int(sizeof(T) / 16);
        uint4 w[n];
#pragma unroll
        for (int k = 0; k < n; ++k) w[k] = __ldcs(reinterpret_cast<const uint4*>(p) + k);
        T v;
        memcpy(&v, w, sizeof(T));
        return v;
    } else {
        static_assert(sizeof(T) % 8 == 0 && alignof(T) >= 8, "path state records are whole 8-byte words");
        constexpr int n = int(sizeof(T) / 8);
        unsigned long long w[n];
#pragma unroll
        for (int k = 0; k < n; ++k) w[k] = __ldcs(reinterpret_cast<const unsigned long long*>(p) + k);
        T v;
        memcpy(&v, w, sizeof(T));
        return v;
    }
#else
    return *p;
#endif
}
template <class T>
__device__ __forceinline__ void storeStream(T* p, const T& v) {
#if OWEC_STREAM_STATE
    if constexpr (alignof(T) >= 16 && sizeof(T) % 16 == 0) {
        constexpr int n = int(sizeof(T) / 16);
        uint4 w[n];
        memcpy(w, &v, sizeof(T));
#pragma unroll
        for (int k = 0; k < n; ++k) __stcs(reinterpret_cast<uint4*>(p) + k, w[k]);
    } else {
        static_assert(sizeof(T) % 8 == 0 && alignof(T) >= 8, "path state records are whole 8-byte words");
        constexpr int n = int(sizeof(T) / 8);
        unsigned long long w[n];
        memcpy(w, &v, sizeof(T));
#pragma unroll
        for (int k = 0; k < n; ++k) __stcs(reinterpret_cast<unsigned long long*>(p) + k, w[k]);
    }
#else
    *p = v;
#endif
}

// A pending next-event visibility query and its contribution if the segment is clear.
template <class R>
struct alignas(16) ShadowRay {
    double o[3];
    R d[3];
    double tmax;          // Inf for the sun
    uint32_t region;      // region the segment starts in
    uint32_t endRegion;   // region it must arrive in (kNone: the ambient region for the sun)
    uint32_t depB, depP;
    uint32_t endB;        // the light's boundary (kNone: the sun, or an eye the ray connects to)
    uint32_t path;
    float errN;
    float contrib[4];     // beta * f * Le * cos * w / pdf, before transmittance
};
static_assert(sizeof(ShadowRay<float>) == 96, "a mixed-precision shadow record stays six 16-byte words");

// Device time of a pass's closest-hit and shadow kernels (owec_last_pass_timing), in nanoseconds of the
// global timer, from a kernel's first thread to its last warp. The two kinds overlap: a bounce's shadow
// kernels run beside the next bounce's closest-hit kernel.
struct BounceClock {
    unsigned long long intersect, shadow;
};

// Counters of one bounce; every bounce of a batch has its own set, all cleared at once before it.
constexpr int kCountActive = 0, kCountSurface = 2, kCountShadow = 3, kFetchIntersect = 4, kFetchShadow = 5, kCountSimple = 6,
              kClockIntersect = 8, kClockShadow = 10,  // 64-bit words (stampStart)
              kBounceCounters = 12, kCountNext = kBounceCounters + kCountActive;
// The paths a bounce started with, as the closest-hit kernel reports them to the host (Queues::progress):
// the bounce's number in the upper half, so that a stale word is never taken for it.
constexpr int kProgressSlots = 64;

struct Queues {
    uint32_t* active[2];      // this bounce's paths and the next one's
    uint32_t* surface;        // surface events with any optics
    uint32_t* shadow;
    uint32_t* counts;         // this bounce's counters, the next bounce's behind them
    uint32_t* surfaceSimple;  // surface events on Lambertian, absorbing and detecting boundaries
    BounceClock* clock;       // null: not timed
    unsigned long long* progress;  // this bounce's word in page-locked host memory
    uint32_t bounce;          // this bounce's number, counted on from pass to pass
};

#if defined(__CUDACC__)
__device__ __forceinline__ unsigned long long globalTimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ bool firstThread() { return blockIdx.x == 0 && threadIdx.x == 0; }
// A kernel's time in one 64-bit word of its bounce's counters: the first thread adds the time it starts at (modulo
// 2^44 ns) above kClockBits, one lane of each warp adds one at the warp's end, and the last one finds the start
// beside the count. One word needs no fence, which cost the FP32 room half a percent of a pass.
constexpr int kClockBits = 20;
__device__ __forceinline__ void stampStart(uint32_t* word) {
    atomicAdd(reinterpret_cast<unsigned long long*>(word), globalTimer() << kClockBits);
}
__device__ __forceinline__ void stampEnd(uint32_t* word, unsigned long long& sum) {
    const unsigned long long before = atomicAdd(reinterpret_cast<unsigned long long*>(word), 1ull);
    if ((before & ((1ull << kClockBits) - 1)) + 1 != gridDim.x * (blockDim.x >> 5)) return;
    sum += (globalTimer() - (before >> kClockBits)) & (~0ull >> kClockBits);
}
// The first thread of a bounce's closest-hit kernel, and of its first shadow kernel.
__device__ __forceinline__ void stampIntersect(const Queues& q) {
    *reinterpret_cast<volatile unsigned long long*>(q.progress) = (uint64_t(q.bounce) << 32) | q.counts[kCountActive];
    if (q.clock) stampStart(q.counts + kClockIntersect);
}
__device__ __forceinline__ void stampShadow(const Queues& q) {
    if (q.clock) stampStart(q.counts + kClockShadow);
}
#endif

struct StatCounters {
    unsigned long long paths, segments, inconsistencies, leaks, shadowRays, faults;
};

template <class R>
struct PathBuffers {
    PathRay<R>* ray;
    PathSpec<R>* spec;
    PathAux* aux;
    HitRec* hit;
    ShadowRay<R>* shadow;  // indexed by shadow-queue position
    float* sampleXyz;      // 3 per path slot: the path's XYZ estimate once the batch is done
};

struct PassParams {
    uint64_t seed;
    int32_t maxDepth, rrDepth;
    int32_t wavelengthMode;
    float lambdaMin, lambdaMax;
    float fresnelFloor;
    uint32_t nPixels;        // detector pixels
    uint32_t nPaths;         // paths in this batch: nPixels * samples
    uint32_t streamBase;     // PCG32 stream of the batch's first sample
    int32_t anyHitShadows;   // 1: no null boundaries, shadow rays stop at the first crossing
    // The adjoint's first phase: a path about to meet boundary ckptBoundary (kNone: never) stops there
    // and leaves its state as a PathCheckpoint (slot from ckptCount) for the derivative replay.
    uint32_t ckptBoundary = kNone;
    uint32_t* ckptCount = nullptr;
    void* ckpt = nullptr;
};

// A path's state at the surface event where it first meets the heightfield: what kSurface would
// load for it (after the free flight of the segment), and the hit.
template <class R>
struct alignas(16) PathCheckpoint {
    PathRay<R> ray;
    PathSpec<R> spec;
    PathAux aux;
    HitRec hit;
};

}  // namespace owec
