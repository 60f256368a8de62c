// Wavefront spectral path tracer with MIS next-event estimation.
//
// Per launch (one or more samples per pixel):
//   cameraTraceKernel camera rays for every path slot (path_tracing.cu:30-77)
//                     and their closest hits
//   per bounce b:
//     traceShadowKernel (from the second bounce on) closest hit of the active
//                     rays, then the path index is appended to the queue of
//                     the hit material's BSDF kind (or the miss queue):
//                     material-sorted shading; and any-hit visibility of the
//                     NEE rays of the bounce before, whose contribution is
//                     added when unoccluded
//     shadeKernel     walks the sorted queues; implicit emission with MIS,
//                     Russian roulette, NEE light sample, BSDF sample
//                     (path_tracing.cu:133-259, miss :266-337); the last
//                     bounce casts no NEE rays
//   filmResolveKernel bins each path's 4-wavelength contribution into 16 FP64
//                     strata of its pixel (spectrum_types.h:674-684) and
//                     converts a finished call's film to colours
// Queue lengths live in device counters, so a launch never synchronises with
// the host and its fixed kernel sequence can be captured in a CUDA graph.
#include "pt.cuh"
#include <cuda_fp16.h>
#include "guide_mlp.cuh"
#include "tables.cuh"
#include "wavefront.cuh"
#include "pt_shade.cuh"

#include <algorithm>
#include <random>
#include <stdexcept>
#include <string>
#include <type_traits>
#include <utility>

namespace vlrb {

namespace {

// The launch's kernels follow one another with programmatic dependent launch:
// once every block of a kernel has started, the next kernel's blocks take the
// slots that fall free and wait here for the kernel before them to end, so a
// launch does not begin with an empty GPU.  Every kernel of the chain waits
// before it touches memory, so the end of one implies the end of all before
// it.  Measured on frames of many short launches: 256 x 256, 1 spp 409 -> 400
// us; small terrain 637 x 359, 4 spp 1.43 -> 1.39 ms; the large ones the same.
//
// Not while capturing: in a graph the programmatic edges keep side-by-side
// branches from sharing the GPU.  Graph of Cornell boxes of 64, 128, 256 and 320
// pixels a side, 8 spp each: 1.74 ms with them, 1.00 without; twelve of 128, 2
// spp: 2.47 and 0.89.  (The same renders on streams of their own: 1.21 and 1.13;
// 1.21 and 1.21.)
__device__ __forceinline__ void startDependent() {
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
}

struct Chain {
    cudaStream_t stream;
    bool programmatic;
    explicit Chain(cudaStream_t s) : stream(s), programmatic(true) {
        if (s == nullptr) return;   // the legacy stream cannot be captured
        cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
        programmatic = cudaStreamIsCapturing(s, &status) == cudaSuccess && status == cudaStreamCaptureStatusNone;
    }
};

template <class... Params, class... Args>
inline void launchChained(void (*kernel)(Params...), uint32_t grid, uint32_t block, const Chain &chain,
                          Args &&...args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.stream = chain.stream;
    cfg.attrs = &attr;
    cfg.numAttrs = chain.programmatic ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
    if (e != cudaSuccess) throw std::runtime_error(std::string("pt launch: ") + cudaGetErrorString(e));
}

// The fields of PathBuffers::meta.
constexpr uint32_t kPrevTypeShift = 25;
__device__ __forceinline__ WLS wlsOf(const uint4 &meta) {
    WLS w;
    w.setOffset(__uint_as_float(meta.w));
    w.selected = meta.x & 0xFu;
    w.single = (meta.x >> 4) & 1u;
    return w;
}

// Threads per block of the ray kernels.  A block keeps its warps' registers
// until its slowest ray is done, so rays run in blocks of two warps (the least
// with which the limit of 32 blocks still fills an SM).  Blocks of 256 / 128 /
// 64: terrain 1920 x 1080, 4 spp, 10.46, 10.30, 10.26 ms; Cornell box 512 x
// 512, 64 spp, 7.60, 7.56, 7.51 ms.  More threads than the shading kernels
// have balance long traversals better but cost the short launches: twice as
// many, terrain 10.09 ms, but a 1-spp 1920 x 1080 Cornell frame 1.64 -> 1.69
// ms; warps that take their rays from a counter, terrain 9.90 ms, but Cornell
// 8.16 ms (one atomic per 32 short rays).
constexpr uint32_t kRayThreads = 64;

// Camera rays of every path slot, traced at once: the camera's work is bound by
// the path state it writes and the traversal by latency, so one hides the
// other, and the ray and its queue entry are not read back (Cornell box, 512 x
// 512, 64 spp: camera 0.35 + trace 2.96 ms apart, 3.15 together).
__global__ void __launch_bounds__(kRayThreads, 20) cameraTraceKernel(SceneGPU S, PathBuffers pb, FrameParams fp) {
    startDependent();
    const uint32_t P = fp.numPaths;
    uint32_t* ctr = bounceCounters(pb, 0);
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < P; p += gridDim.x * blockDim.x) {
        const uint32_t pixel = pixelOfPath(p, fp.width, fp.height);
        PCG32 rng{ pb.rng[p] };
        const CameraRay cr = cameraSample(S, pixel % fp.width, pixel / fp.width, fp.width, fp.height, rng);
        pb.rng[p] = rng.state;
        pb.meta[p] = make_uint4(cr.wls.selected | ((dir::Acquisition | dir::LowFreq) << kPrevTypeShift),
                                __float_as_uint(cr.initImportance), __float_as_uint(cr.dirPDF),
                                __float_as_uint(cr.wavelengthOffset));
        pb.alpha[p] = toF4(cr.alpha);
        pb.contrib[p] = make_float4(0.f, 0.f, 0.f, 0.f);
        pb.rayOrg[p] = make_float4(cr.org.x, cr.org.y, cr.org.z, FLT_MAX);
        pb.rayDir[p] = make_float4(cr.dir.x, cr.dir.y, cr.dir.z, 0.0f);
        traceFrom(S, pb, P, ctr, p, cr.org, cr.dir, FLT_MAX);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) ctr[kCntActive] = P;
}

// Visibility of one NEE ray; adds its contribution when unoccluded.
__device__ __forceinline__ void traceShadow(const SceneGPU &S, const PathBuffers &pb, uint32_t i) {
    ShadowRay sr = pb.shadow[i];
    const float vis = shadowVisibility(S, V3(sr.org.x, sr.org.y, sr.org.z), V3(sr.dir.x, sr.dir.y, sr.dir.z),
                                       sr.org.w);
    if (vis != 0.0f) {
        uint32_t p = __float_as_uint(sr.dir.w);
        float4 c = pb.contrib[p];
        c.x += vis * sr.contrib.x; c.y += vis * sr.contrib.y; c.z += vis * sr.contrib.z; c.w += vis * sr.contrib.w;
        pb.contrib[p] = c;
    }
}

__global__ void __launch_bounds__(256, 5) traceKernel(SceneGPU S, PathBuffers pb, FrameParams fp) {
    uint32_t* ctr = bounceCounters(pb, fp.bounce);
    const uint32_t n = ctr[kCntActive];
    const uint32_t* queue = pb.active[fp.bounce & 1];
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        tracePath(S, pb, fp.numPaths, ctr, queue[i]);
}

// The rays of one shade pass in one launch: the extension rays of bounce
// fp.bounce and the shadow rays of the bounce before it (a warp holds rays of
// one type).  Both are bound by latency and divergence and each ends in a
// long tail of a few slow rays, so running them together fills the one's
// idle slots with the other's rays: terrain scene of 3.4 M triangles, 1920 x
// 1080, 4 spp, 12 bounces, trace + shadow 9.80 ms as two launches a bounce,
// 8.70 together, 8.35 at 48 warps per SM (40 registers), 8.10 in blocks of
// kRayThreads.
__global__ void __launch_bounds__(kRayThreads, 24) traceShadowKernel(SceneGPU S, PathBuffers pb, FrameParams fp) {
    startDependent();
    uint32_t* ctr = bounceCounters(pb, fp.bounce);
    const uint32_t n = ctr[kCntActive], m = bounceCounters(pb, fp.bounce - 1)[kCntShadow];
    const uint32_t nWarps = (n + 31) & ~31u;   // a warp holds rays of one type
    const uint32_t* queue = pb.active[fp.bounce & 1];
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nWarps + m; i += gridDim.x * blockDim.x) {
        if (i >= nWarps) traceShadow(S, pb, i - nWarps);
        else if (i < n) tracePath(S, pb, fp.numPaths, ctr, queue[i]);
    }
}

__device__ __forceinline__ float4* recField(const GuideFrame &gf, uint32_t P, uint32_t b, uint32_t f) {
    return gf.rec + (static_cast<size_t>(b) * kRecFields + f) * P;
}

// Completes the training record of the previous bounce with the path's
// contribution so far (everything gathered after the snapshot is the
// indirect light the previous vertex received along its sampled direction).
__device__ __forceinline__ void completeRecord(const GuideFrame &gf, uint32_t P, uint32_t bounce, uint32_t p,
                                               uint32_t flags, const S4 &contrib) {
    if (!(flags & kFlagRecordPending) || bounce == 0) return;
    const uint32_t b = bounce - 1;
    recField(gf, P, b, 5)[p] = toF4(contrib);
    gf.recStamp[static_cast<size_t>(b) * P + p] = gf.counts[kCountStamp];
}

__device__ __forceinline__ uint32_t packHalf2(float a, float b) {
    __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ float2 unpackHalf2(uint32_t u) {
    return __half22float2(*reinterpret_cast<const __half2*>(&u));
}

// The stored mixture (112 B per path): directions, concentrations and
// weights in half precision, and per lobe the FP32 factor that turns
// exp(kappa (mu.w - 1)) into density, computed from the rounded values the
// sampler uses, so sampling and pdf stay one density.
__device__ __forceinline__ void loadMixture(const GuideFrame &gf, uint32_t P, uint32_t p, guide::Mixture &m) {
#pragma unroll
    for (int k = 0; k < guide::kLobes; ++k) {
        const uint2 q = gf.lobes[static_cast<size_t>(k) * P + p];
        const float2 a = unpackHalf2(q.x), b = unpackHalf2(q.y);
        const float inv = rsqrtf(a.x * a.x + a.y * a.y + b.x * b.x);
        m.lobe[k] = make_float4(a.x * inv, a.y * inv, b.x * inv, b.y);
    }
    const uint2 w0 = gf.lobeWeights[p], w1 = gf.lobeWeights[static_cast<size_t>(P) + p];
    const float2 a = unpackHalf2(w0.x), b = unpackHalf2(w0.y), c = unpackHalf2(w1.x), d = unpackHalf2(w1.y);
    m.weight[0] = a.x; m.weight[1] = a.y; m.weight[2] = b.x; m.weight[3] = b.y;
    m.weight[4] = c.x; m.weight[5] = c.y; m.weight[6] = d.x; m.weight[7] = d.y;
    const float4 s0 = gf.lobeScales[p], s1 = gf.lobeScales[static_cast<size_t>(P) + p];
    m.scale[0] = s0.x; m.scale[1] = s0.y; m.scale[2] = s0.z; m.scale[3] = s0.w;
    m.scale[4] = s1.x; m.scale[5] = s1.y; m.scale[6] = s1.z; m.scale[7] = s1.w;
}

// Bound by latency: a hit is a chain of gathers (queue entry, path state, the
// triangle's line, material, spectra, light) and about 2,000 instructions a
// warp, with 24 warps per SM (80 registers).  What was taken out of the chain:
// the path's flags, importances, previous sample and wavelengths are one
// 16-byte record, the triangle one 128-byte line, its contribution is read and
// written only where light is added and the ray's origin only at emitters.
// Cornell box, 512 x 512, 64 spp: 5.51 -> 4.42 ms a frame; terrain, 1920 x 1080,
// 4 spp: 2.66 -> 2.22 ms.  Measured and not
// kept: the next path's state prefetched into L1 or L2 (5.02 ms), blocks of
// 128 threads with 6, 7 or 8 per SM (4.78, 4.87, 4.96 ms).
template <bool kGuide, bool kMaps>
__global__ void __launch_bounds__(256, 3) shadeKernel(SceneGPU S, PathBuffers pb, FrameParams fp, GuideFrame gf) {
    startDependent();
    uint32_t* ctr = bounceCounters(pb, fp.bounce);
    uint32_t* next = bounceCounters(pb, fp.bounce + 1);
    __shared__ uint32_t sOff[kNumShadeBuckets + 1];
    if (threadIdx.x == 0) {
        uint32_t run = 0;
        for (uint32_t k = 0; k < kNumShadeBuckets; ++k) { sOff[k] = run; run += ctr[kCntBucket0 + k]; }
        sOff[kNumShadeBuckets] = run;
    }
    __syncthreads();
    const uint32_t total = sOff[kNumShadeBuckets];
    const uint32_t P = fp.numPaths;
    uint32_t* nextQueue = pb.active[(fp.bounce + 1) & 1];
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < total; j += gridDim.x * blockDim.x) {
        uint32_t k = 0;
        while (j >= sOff[k + 1]) ++k;
        const uint32_t p = pb.buckets[k * P + (j - sOff[k])];
        const uint4 meta = pb.meta[p];
        const WLS wls = wlsOf(meta);
        uint32_t flags = meta.x;
        const PrevInRegisters prev{ meta.x >> kPrevTypeShift, __uint_as_float(meta.z) };
        uint32_t pathLength = ((flags >> 8) & 0xFFFFu) + 1;
        bool maxLengthTerminate = pathLength >= fp.maxPathLength;
        const uint32_t flagsIn = flags;
        flags = (flags & 0x1Fu) | (pathLength << 8) | (maxLengthTerminate ? 0x20u : 0u);
        // The path's contribution is touched only where something is added
        // to it (a light, the environment) or a training record reads it.
        const bool closesRecord = kGuide && (flagsIn & kFlagRecordPending) && fp.bounce > 0;
        if (k == kNumBsdfKinds) {
            if (S.envInst >= 0 || closesRecord) {
                S4 contrib = toS4(pb.contrib[p]);
                const float4 d4 = pb.rayDir[p];
                envMissContribution(S, V3(d4.x, d4.y, d4.z), wls, toS4(pb.alpha[p]), prev, pathLength, contrib);
                if constexpr (kGuide) completeRecord(gf, P, fp.bounce, p, flagsIn, contrib);
                pb.contrib[p] = toF4(contrib);
            }
            continue;
        }
        float4 h = pb.hit[p];
        const uint32_t prim = __float_as_uint(h.w);
        SurfPt sp;
        float area;
        decodeHit<kMaps>(S, prim, h.y, h.z, &sp, &area);
        const uint32_t matIndex = sp.material;
        const MatDesc &mat = S.mats[matIndex];
        float bsdfScale = 1.0f;
        const uint32_t bsdfIndex =
            mat.bsdfKind == kMultiBSDF ? bsdfMaterial(S, matIndex, pb.rng[p], prim, &bsdfScale) : matIndex;
        Bsdf bsdf = buildBsdf<-1, kMaps>(S.meng, S.mats[bsdfIndex], wls, sp.tu, sp.tv);
        const float4 d4 = pb.rayDir[p];
        const V3 rayDir(d4.x, d4.y, d4.z);
        V3 dirOutLocal = sp.frame.toLocal(-rayDir);
        S4 alpha = toS4(pb.alpha[p]);
        // implicit light sampling
        if (mat.emitter != kEmitNone || closesRecord) {
            S4 contrib = toS4(pb.contrib[p]);
            const float4 o4 = pb.rayOrg[p];
            implicitEmission(S, mat, wls, sp, dirOutLocal, V3(o4.x, o4.y, o4.z), area, prev, pathLength, alpha, contrib);
            // The record of the previous vertex closes after this vertex's
            // emission: light reached directly from there is NEE's job, and
            // the network learns the indirect light NEE cannot sample.
            if constexpr (kGuide) completeRecord(gf, P, fp.bounce, p, flagsIn, contrib);
            pb.contrib[p] = toF4(contrib);
        }
        alpha *= bsdfScale;   // a Multi material's component choice (after the emission)
        if (maxLengthTerminate) continue;
        PCG32 rng{ pb.rng[p] };
        // Russian roulette on the hero-weighted throughput
        float continueProb = fminf(alpha.importance(wls.selected) / __uint_as_float(meta.y), 1.0f);
        if (rng.uniform() >= continueProb) { pb.rng[p] = rng.state; continue; }
        alpha /= continueProb;
        V3 gnLocal = sp.frame.toLocal(sp.gn);
        BsdfQuery q;
        q.dirLocal = dirOutLocal;
        q.wlHint = wls.selected;
        q.filter = dir::All;
        q.importanceMode = 0;
        bool guided = false;
        guide::Mixture mix;
        if constexpr (kGuide) {
            guided = gf.sample && isGuidedKind(k) && fp.bounce < gf.recBounces;
            if (guided) loadMixture(gf, P, p, mix);
        }
        // next-event estimation
        {
            NeeRay nr;
            if (neeSample<kGuide>(S, sp, bsdf, q, gnLocal, wls, alpha, rng, guided, mix, &nr)) {
                uint32_t slot = appendSlot(ctr + kCntShadow, 0u);
                ShadowRay sr;
                sr.org = make_float4(nr.org.x, nr.org.y, nr.org.z, nr.tmax);
                sr.dir = make_float4(nr.dir.x, nr.dir.y, nr.dir.z, __uint_as_float(p));
                sr.contrib = toF4(nr.contrib);
                pb.shadow[slot] = sr;
            }
        }
        // BSDF sampling (guided kinds: one-sample MIS of BSDF and mixture)
        float uc = rng.uniform(), ud0 = rng.uniform(), ud1 = rng.uniform();
        BsdfSample bs;
        S4 fs;
        if constexpr (kGuide) {
            if (guided) {
                const float uSel = rng.uniform();
                V3 wiW;
                float pB;
                if (uSel < 0.5f) {
                    wiW = guide::mixtureSample(mix, uc, ud0, ud1);
                    bs.dirLocal = sp.frame.toLocal(wiW);
                    fs = bsdfEval(bsdf, q, gnLocal, bs.dirLocal, nullptr);
                    pB = bsdfPDF(bsdf, q, bs.dirLocal, nullptr);
                    bs.sampledType = dir::LowFreq | (dot(bs.dirLocal, gnLocal) > 0.0f ? dir::Reflection
                                                                                       : dir::Transmission);
                }
                else {
                    fs = bsdfSample(bsdf, q, gnLocal, uc, ud0, ud1, &bs, nullptr);
                    pB = bs.dirPDF;
                    wiW = sp.frame.fromLocal(bs.dirLocal);
                }
                bs.dirPDF = 0.5f * pB + 0.5f * guide::mixturePdf(mix, wiW);
            }
            else fs = bsdfSample(bsdf, q, gnLocal, uc, ud0, ud1, &bs, nullptr);
        }
        else fs = bsdfSample(bsdf, q, gnLocal, uc, ud0, ud1, &bs, nullptr);
        pb.rng[p] = rng.state;
        if (fs.isZero() || !(bs.dirPDF > 0.0f)) continue;
        if (dir::isDispersive(bs.sampledType) && !wls.single) {
            bs.dirPDF /= kNumLambdas;
            flags |= 0x10u;
        }
        float cosFactor = dot(bs.dirLocal, gnLocal);
        V3 dirIn = sp.frame.fromLocal(bs.dirLocal);
        if constexpr (kGuide) {
            if (gf.record && fp.bounce < gf.recBounces && isGuidedKind(k)) {
                recField(gf, P, fp.bounce, 0)[p] = make_float4(sp.position.x, sp.position.y, sp.position.z, 0.0f);
                recField(gf, P, fp.bounce, 1)[p] = make_float4(sp.frame.z.x, sp.frame.z.y, sp.frame.z.z, 0.0f);
                recField(gf, P, fp.bounce, 2)[p] = make_float4(-rayDir.x, -rayDir.y, -rayDir.z, 0.0f);
                recField(gf, P, fp.bounce, 3)[p] = make_float4(dirIn.x, dirIn.y, dirIn.z, 0.0f);
                recField(gf, P, fp.bounce, 4)[p] = toF4(alpha);
                flags |= kFlagRecordPending;
            }
        }
        alpha *= fs * (fabsf(cosFactor) / bs.dirPDF);
        V3 org = offsetRayOrigin(sp.position, cosFactor > 0.0f ? sp.gn : -sp.gn);
        pb.alpha[p] = toF4(alpha);
        pb.meta[p] = make_uint4(flags | (bs.sampledType << kPrevTypeShift), meta.y, __float_as_uint(bs.dirPDF), meta.w);
        pb.rayOrg[p] = make_float4(org.x, org.y, org.z, FLT_MAX);
        pb.rayDir[p] = make_float4(dirIn.x, dirIn.y, dirIn.z, 0.0f);
        uint32_t slot = appendSlot(next + kCntActive, 0u);
        nextQueue[slot] = p;
    }
}

// ---- learned guiding: network queries straight from the sorted hit queues
struct GuidedHitSrc {
    SceneGPU S;
    PathBuffers pb;
    FrameParams fp;
    guide::Net net;
    __device__ void counts(uint32_t c[3]) const {
        const uint32_t* ctr = bounceCounters(pb, fp.bounce);
        c[0] = ctr[kCntBucket0 + kMatte];
        c[1] = ctr[kCntBucket0 + kLambertianBSDF];
        c[2] = ctr[kCntBucket0 + kUE4];
    }
    __device__ uint32_t count() const {
        uint32_t c[3];
        counts(c);
        return c[0] + c[1] + c[2];
    }
    __device__ uint32_t pathOf(uint32_t i) const {
        uint32_t c[3];
        counts(c);
        uint32_t k = kMatte;
        if (i >= c[0]) { i -= c[0]; k = kLambertianBSDF; if (i >= c[1]) { i -= c[1]; k = kUE4; } }
        return pb.buckets[k * fp.numPaths + i];
    }
    __device__ bool load(uint32_t i, float3* p01, V3* wo, V3* nrm) const {
        const uint32_t p = pathOf(i);
        const float4 h = pb.hit[p];
        SurfPt sp;
        decodeHit(S, __float_as_uint(h.w), h.y, h.z, &sp, nullptr);
        const float4 d = pb.rayDir[p];
        *p01 = guide::normalisedPosition(net, sp.position.x, sp.position.y, sp.position.z);
        *wo = V3(-d.x, -d.y, -d.z);
        *nrm = sp.frame.z;
        return true;
    }
};

struct MixtureDst {
    GuidedHitSrc src;
    uint2* lobes;
    uint2* lobeWeights;
    float4* lobeScales;
    __device__ void store(uint32_t i, const float y[guide::kOut]) const {
        const uint32_t p = src.pathOf(i);
        const uint32_t P = src.fp.numPaths;
        guide::Mixture m;
        guide::decodeMixture(y, m);
        // round to half, then derive the density factors from what the
        // sampler will read back: lobe k is chosen with the probability its
        // cumulative-weight test gives (the last lobe takes the remainder)
        float w[guide::kLobes], kap[guide::kLobes];
        float acc = 0.0f, prev = 0.0f;
#pragma unroll
        for (int k = 0; k < guide::kLobes; ++k) {
            const float4 l = m.lobe[k];
            lobes[static_cast<size_t>(k) * P + p] = make_uint2(packHalf2(l.x, l.y), packHalf2(l.z, l.w));
            kap[k] = unpackHalf2(packHalf2(l.w, 0.0f)).x;
            w[k] = unpackHalf2(packHalf2(m.weight[k], 0.0f)).x;
        }
        lobeWeights[p] = make_uint2(packHalf2(w[0], w[1]), packHalf2(w[2], w[3]));
        lobeWeights[static_cast<size_t>(P) + p] = make_uint2(packHalf2(w[4], w[5]), packHalf2(w[6], w[7]));
        float sc[guide::kLobes];
#pragma unroll
        for (int k = 0; k < guide::kLobes; ++k) {
            acc += w[k];
            const float cum = k == guide::kLobes - 1 ? 1.0f : fminf(acc, 1.0f);
            const float prob = fmaxf(cum - prev, 0.0f);
            prev = fmaxf(prev, cum);
            sc[k] = prob * expf(guide::vmfLogNorm(kap[k]));
        }
        lobeScales[p] = make_float4(sc[0], sc[1], sc[2], sc[3]);
        lobeScales[static_cast<size_t>(P) + p] = make_float4(sc[4], sc[5], sc[6], sc[7]);
    }
};

__device__ __forceinline__ uint32_t mixBits(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t h = a * 0x9E3779B1u ^ (b + 0x7F4A7C15u) * 0x85EBCA77u ^ c * 0xC2B2AE3Du;
    h ^= h >> 15; h *= 0x2C1B3C6Du; h ^= h >> 12; h *= 0x297A2D39u; h ^= h >> 15;
    return h;
}

// Turns the launch's complete records into training samples: weight =
// mean over the 4 wavelengths of (contribution gathered after the vertex) /
// (throughput at the vertex), i.e. incident radiance x BSDF x cos / pdf of the
// sampled direction.  A random subset of about targetSamples is kept.
__global__ void __launch_bounds__(256) guideFinalizeKernel(PathBuffers pb, FrameParams fp, GuideFrame gf) {
    const uint32_t P = fp.numPaths;
    const uint32_t last = gf.counts[2];
    const uint32_t stamp = gf.counts[kCountStamp];
    const float accept = last > gf.targetSamples ? static_cast<float>(gf.targetSamples) / last : 1.0f;
    // one thread per (bounce, path) record: independent loads in flight
    const size_t total = static_cast<size_t>(P) * gf.recBounces;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const uint32_t b = static_cast<uint32_t>(i / P), p = static_cast<uint32_t>(i % P);
        {
            float w = 0.0f;
            if (gf.recStamp[i] == stamp) {
                const float4 cEnd = pb.contrib[p];
                const float4 beta = recField(gf, P, b, 4)[p];
                const float4 snap = recField(gf, P, b, 5)[p];
                const float bt[4] = { beta.x, beta.y, beta.z, beta.w };
                const float dc[4] = { cEnd.x - snap.x, cEnd.y - snap.y, cEnd.z - snap.z, cEnd.w - snap.w };
                for (int i = 0; i < 4; ++i)
                    if (bt[i] > 0.0f) w += fmaxf(dc[i], 0.0f) / bt[i];
                w *= 0.25f;
            }
            const bool cand = w > 0.0f && isfinite(w);
            const bool keep = cand && (mixBits(p, b, stamp) >> 8) * (1.0f / 16777216.0f) < accept;
            // one atomic per warp for the candidate count and the slots
            const uint32_t active = __activemask();
            const int leader = __ffs(active) - 1;
            const uint32_t lane = threadIdx.x & 31;
            const uint32_t cm = __ballot_sync(active, cand), km = __ballot_sync(active, keep);
            uint32_t base = 0;
            if (static_cast<int>(lane) == leader) {
                if (cm) atomicAdd(gf.counts + 1, static_cast<uint32_t>(__popc(cm)));
                if (km) base = atomicAdd(gf.counts, static_cast<uint32_t>(__popc(km)));
            }
            base = __shfl_sync(active, base, leader);
            const uint32_t slot = base + __popc(km & ((1u << lane) - 1u));
            if (!keep || slot >= gf.sampleCapacity) continue;
            const float4 pos = recField(gf, P, b, 0)[p];
            guide::Sample smp;
            smp.posWeight = make_float4(pos.x, pos.y, pos.z, w);
            smp.nrm = recField(gf, P, b, 1)[p];
            smp.wo = recField(gf, P, b, 2)[p];
            smp.wi = recField(gf, P, b, 3)[p];
            gf.samples[slot] = smp;
        }
    }
}

// Start of a recording launch: accepted = 0, last = this, this = 0, next
// stamp.  All on the device, so a captured launch sequence replays correctly.
__global__ void guideCountsKernel(uint32_t* counts) {
    counts[2] = counts[1] > 0 ? counts[1] : counts[2];
    counts[1] = 0;
    counts[0] = 0;
    counts[kCountStamp] += 1;
}

struct FilmConst {
    float xbar[kNumStrata], ybar[kNumStrata], zbar[kNumStrata];
    float integralCMF;
    float xyzToRgb[9];
};

__device__ __forceinline__ float4 strataToRGBA(const double* s, const FilmConst &fc, uint32_t n, uint32_t frames) {
    double X = 0, Y = 0, Z = 0;
    for (uint32_t k = 0; k < kNumStrata; ++k) {
        double v = s[k];
        X += fc.xbar[k] * v;
        Y += fc.ybar[k] * v;
        Z += fc.zbar[k] * v;
    }
    double scale = static_cast<double>(n) / (static_cast<double>(fc.integralCMF) * frames);
    float xyz[3] = { static_cast<float>(X * scale), static_cast<float>(Y * scale), static_cast<float>(Z * scale) };
    float rgb[3];
    mulColMajor(fc.xyzToRgb, xyz, rgb);
    return make_float4(rgb[0], rgb[1], rgb[2], 1.0f);
}

__global__ void filmAddFramesKernel(uint32_t* frames, uint32_t samples) { *frames += samples; }

__global__ void filmToRGBAKernel(Film film, FilmConst fc, float4* out) {
    const uint32_t n = film.width * film.height;
    const uint32_t frames = *film.frames ? *film.frames : 1u;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        out[i] = strataToRGBA(film.strata + static_cast<size_t>(i) * kNumStrata, fc, n, frames);
    }
}

// The launch's contributions into the film.  `lanes` threads (a power of two
// up to 32) share a pixel: each bins every lanes-th of its samples (path slots
// pixelCount apart) into 16 FP64 strata of its own in shared memory, four
// samples' loads at a time, and the warp then adds its pixels' strata, the
// lanes' sums in order, to the film in whole lines.  The pixels have one
// writer, so there are no atomics.  `overwrite`: the first launch of an
// accumulation stores instead of adding (no clear, no read).  `out`: the
// pixel's colour from the strata just written, XYZ / frames * (W*H) -> Rec.709
// D65, with `samples` added to the device frame count (the last launch of a
// call that renders the whole film).
//
// Bound by HBM where the pixels fill the GPU: 32 B read per sample, 128 B
// written (and read when adding) per pixel, 16 B of colour.  With fewer pixels
// a thread's samples are the chain, so the pixels are split (filmLanes).  With
// one thread a pixel, one sample at a time, and now: 64 x 64 pixels, 512 samples a
// launch, 633 -> 49 us; 32 x 32, 64: 62 -> 17; 512 x 512, 64: 199 -> 136; 1920 x
// 1080, 1, adding to a film: 154 -> 114 (with its lines read ahead of the stores).
// kPitch (odd) spreads the strata over the banks.
constexpr int kFilmThreads = 128, kFilmPitch = kNumStrata + 1;

__device__ __forceinline__ void binSample(double* strata, const float4 &contrib, float offset) {
    const S4 c = toS4(contrib);
    if (!c.allFinite()) return;
    WLS wls;
    wls.setOffset(offset);
#pragma unroll
    for (int w = 0; w < 4; ++w) strata[strataBin(wls.lambda[w])] += strataValue(c[w]);
}

template <bool kSplit, int kLoads, bool kAdd>
__global__ void __launch_bounds__(kFilmThreads) filmResolveKernel(PathBuffers pb, Film film, FrameParams fp,
                                                                  FilmConst fc, FilmResolve fr, uint32_t samples,
                                                                  uint32_t lanesArg) {
    __shared__ double sAcc[kFilmThreads * kFilmPitch];
    startDependent();
    const uint32_t lanes = kSplit ? lanesArg : 1u;
    const uint32_t pixels = fp.width * fp.height;
    const uint32_t lane = threadIdx.x & 31u, sub = lane % lanes;
    const uint32_t warpPixels = 32u / lanes, blockPixels = kFilmThreads / lanes;
    double* mine = sAcc + threadIdx.x * kFilmPitch;
    double* warpAcc = sAcc + (threadIdx.x - lane) * kFilmPitch;
    for (uint32_t base = blockIdx.x * blockPixels; base < pixels; base += gridDim.x * blockPixels) {
        const uint32_t i = base + threadIdx.x / lanes;
        const bool in = i < pixels;
        uint32_t fi = 0;
#pragma unroll
        for (uint32_t k = 0; k < kNumStrata; ++k) mine[k] = 0.0;
        if (in) {
            const uint32_t pixel = pixelOfPath(i, fp.width, fp.height);
            fi = (pixel / fp.width) * fp.stride + pixel % fp.width;
            uint32_t s = sub;
            for (; kLoads > 1 && s + (kLoads - 1) * lanes < samples; s += kLoads * lanes) {
                float4 c[kLoads];
                float offset[kLoads];
#pragma unroll
                for (uint32_t u = 0; u < kLoads; ++u) {
                    const uint32_t p = i + (s + u * lanes) * pixels;
                    c[u] = pb.contrib[p];
                    offset[u] = __uint_as_float(pb.meta[p].w);
                }
#pragma unroll
                for (uint32_t u = 0; u < kLoads; ++u) binSample(mine, c[u], offset[u]);
            }
            for (; s < samples; s += lanes) {
                const uint32_t p = i + s * pixels;
                binSample(mine, pb.contrib[p], __uint_as_float(pb.meta[p].w));
            }
        }
        __syncwarp();
        // two pixels' lines per step; what the film holds is read ahead of the stores
        const uint32_t warpBase = base + (threadIdx.x - lane) / lanes;
        constexpr uint32_t kSteps = kSplit ? 8 : 16;
        auto line = [&](uint32_t r) -> double* {
            const uint32_t j = 2 * r + (lane >> 4);
            const uint32_t fj = __shfl_sync(0xFFFFFFFFu, fi, (j * lanes) & 31u);
            return j < warpPixels && warpBase + j < pixels
                       ? film.strata + static_cast<size_t>(fj) * kNumStrata + (lane & 15u) : nullptr;
        };
        double held[kSteps];
        if (kAdd) {
#pragma unroll
            for (uint32_t r = 0; r < kSteps; ++r) {
                const double* src = line(r);
                held[r] = src ? *src : 0.0;
            }
        }
#pragma unroll
        for (uint32_t r = 0; r < kSteps; ++r) {
            double* dst = line(r);
            if (!dst) continue;
            double* sum = warpAcc + (2 * r + (lane >> 4)) * lanes * kFilmPitch + (lane & 15u);
            double v = *sum;
            if (kSplit)
                for (uint32_t l = 1; l < lanes; ++l) v += sum[l * kFilmPitch];
            if (kAdd) v += held[r];
            if (kSplit || kAdd) *sum = v;
            *dst = v;
        }
        __syncwarp();
        if (in && sub == 0 && fr.out) {
            const uint32_t frames = (fr.overwriteFrames ? 0u : *film.frames) + fr.samples;
            fr.out[fi] = strataToRGBA(mine, fc, film.width * film.height, frames ? frames : 1u);
        }
        __syncwarp();
    }
}

// Threads per pixel of the film pass: as many as fill the GPU (eight blocks an
// SM), with four samples' loads in flight each (256 x 256, 4 samples: 17 us with
// one thread a pixel, 23 with four).
inline uint32_t filmLanes(uint32_t pixels, uint32_t samples, int numSMs) {
    const uint64_t wanted = static_cast<uint64_t>(numSMs) * 8 * kFilmThreads;
    uint32_t lanes = 1;
    while (lanes < 32 && 8 * lanes <= samples && static_cast<uint64_t>(pixels) * lanes < wanted) lanes *= 2;
    return lanes;
}

// Adds this launch's per-bounce queue lengths to the running totals, and a
// resolved call's samples to the film's frame count.
__global__ void statsKernel(PathBuffers pb, uint32_t bounces, uint32_t* frames, FilmResolve fr) {
    startDependent();
    unsigned long long seg = 0, sh = 0;
    for (uint32_t b = threadIdx.x; b < bounces; b += 32) {
        seg += bounceCounters(pb, b)[kCntActive];
        sh += bounceCounters(pb, b)[kCntShadow];
    }
    for (int off = 16; off > 0; off >>= 1) {
        seg += __shfl_xor_sync(0xFFFFFFFFu, seg, off);
        sh += __shfl_xor_sync(0xFFFFFFFFu, sh, off);
    }
    if (threadIdx.x == 0) {
        pb.totals[0] += seg;
        pb.totals[1] += sh;
        if (fr.out) *frames = (fr.overwriteFrames ? 0u : *frames) + fr.samples;
    }
}

inline void ck(cudaError_t e, const char* what) {
    if (e != cudaSuccess) throw std::runtime_error(std::string("pt ") + what + ": " + cudaGetErrorString(e));
}

inline size_t a256(size_t x) { return (x + 255) & ~size_t(255); }

} // namespace

size_t pathBufferBytes(uint32_t P, bool wavelengths) {
    size_t b = 0;
    b += a256(size_t(P) * 8);                 // rng
    b += a256(size_t(P) * 16) * (wavelengths ? 2 : 1);   // lambda, alpha
    b += a256(size_t(P) * 4) * 4;             // flags, initImportance, prevDirPDF, prevType
    b += a256(size_t(P) * 16) * 4;            // contrib, rayOrg, rayDir, hit
    b += a256(size_t(P) * 4) * 2;             // active queues
    b += a256(size_t(P) * 4 * kNumShadeBuckets);
    b += a256(size_t(P) * sizeof(ShadowRay));
    b += a256(size_t(kMaxBounces + 1) * kCountersPerBounce * 4);
    b += a256(16);
    return b;
}

void carvePathBuffers(void* base, uint32_t P, PathBuffers* pb, bool wavelengths) {
    char* s = static_cast<char*>(base);
    auto take = [&](size_t bytes) { char* r = s; s += a256(bytes); return r; };
    pb->rng = reinterpret_cast<uint64_t*>(take(size_t(P) * 8));
    pb->lambda = wavelengths ? reinterpret_cast<float4*>(take(size_t(P) * 16)) : nullptr;
    pb->alpha = reinterpret_cast<float4*>(take(size_t(P) * 16));
    pb->meta = reinterpret_cast<uint4*>(s);
    pb->flags = reinterpret_cast<uint32_t*>(take(size_t(P) * 4));
    pb->initImportance = reinterpret_cast<float*>(take(size_t(P) * 4));
    pb->prevDirPDF = reinterpret_cast<float*>(take(size_t(P) * 4));
    pb->prevType = reinterpret_cast<uint32_t*>(take(size_t(P) * 4));
    pb->contrib = reinterpret_cast<float4*>(take(size_t(P) * 16));
    pb->rayOrg = reinterpret_cast<float4*>(take(size_t(P) * 16));
    pb->rayDir = reinterpret_cast<float4*>(take(size_t(P) * 16));
    pb->hit = reinterpret_cast<float4*>(take(size_t(P) * 16));
    pb->active[0] = reinterpret_cast<uint32_t*>(take(size_t(P) * 4));
    pb->active[1] = reinterpret_cast<uint32_t*>(take(size_t(P) * 4));
    pb->buckets = reinterpret_cast<uint32_t*>(take(size_t(P) * 4 * kNumShadeBuckets));
    pb->shadow = reinterpret_cast<ShadowRay*>(take(size_t(P) * sizeof(ShadowRay)));
    pb->counters = reinterpret_cast<uint32_t*>(take(size_t(kMaxBounces + 1) * kCountersPerBounce * 4));
    pb->totals = reinterpret_cast<unsigned long long*>(take(16));
}

size_t guideBufferBytes(uint32_t P, uint32_t recBounces, uint32_t sampleCapacity) {
    size_t b = 0;
    b += a256(size_t(P) * 8 * guide::kLobes);
    b += a256(size_t(P) * 8 * 2) + a256(size_t(P) * 16 * 2);
    b += a256(size_t(P) * 16 * kRecFields * recBounces);
    b += a256(size_t(P) * 4 * recBounces);
    b += a256(size_t(sampleCapacity) * sizeof(guide::Sample));
    b += a256(64);
    return b;
}

void carveGuideBuffers(void* base, uint32_t P, uint32_t recBounces, uint32_t sampleCapacity, GuideFrame* gf) {
    char* s = static_cast<char*>(base);
    auto take = [&](size_t bytes) { char* r = s; s += a256(bytes); return r; };
    gf->lobes = reinterpret_cast<uint2*>(take(size_t(P) * 8 * guide::kLobes));
    gf->lobeWeights = reinterpret_cast<uint2*>(take(size_t(P) * 8 * 2));
    gf->lobeScales = reinterpret_cast<float4*>(take(size_t(P) * 16 * 2));
    gf->rec = reinterpret_cast<float4*>(take(size_t(P) * 16 * kRecFields * recBounces));
    gf->recStamp = reinterpret_cast<uint32_t*>(take(size_t(P) * 4 * recBounces));
    gf->samples = reinterpret_cast<guide::Sample*>(take(size_t(sampleCapacity) * sizeof(guide::Sample)));
    gf->counts = reinterpret_cast<uint32_t*>(take(64));
    gf->err = gf->counts + 8;
    gf->recBounces = recBounces;
    gf->sampleCapacity = sampleCapacity;
}

void seedPathRngs(uint64_t* states, uint32_t n, uint64_t seed) {
    std::mt19937_64 gen(seed);
    for (uint32_t i = 0; i < n; ++i) states[i] = gen();
}

void StageTimer::begin(uint32_t stage, cudaStream_t s, size_t params) {
    ++totalLaunches;
    paramBytes += params;
    if (!enabled) return;
    if (used == kSlots) collect();   // every slot recorded: drain before reuse
    if (used == 0)
        for (auto &e : ev) if (!e) cudaEventCreate(&e);
    stageOf[used] = stage;
    cudaEventRecord(ev[2 * used], s);
}

void StageTimer::end(cudaStream_t s) {
    if (!enabled) return;
    cudaEventRecord(ev[2 * used + 1], s);
    ++used;
}

StageTimer::~StageTimer() {
    for (auto &e : ev) if (e) cudaEventDestroy(e);
}

void StageTimer::collect() {
    if (!enabled) return;
    for (uint32_t i = 0; i < used; ++i) {
        float t = 0.0f;
        cudaEventSynchronize(ev[2 * i + 1]);
        cudaEventElapsedTime(&t, ev[2 * i], ev[2 * i + 1]);
        ms[stageOf[i]] += t;
        launches[stageOf[i]] += 1;
    }
    used = 0;
}

static FilmConst filmConst() {
    FilmConst fc;
    const CmfStrata &cs = hostCmfStrata();
    for (uint32_t k = 0; k < kNumStrata; ++k) { fc.xbar[k] = cs.xbar[k]; fc.ybar[k] = cs.ybar[k]; fc.zbar[k] = cs.zbar[k]; }
    fc.integralCMF = cs.integralCMF;
    for (int k = 0; k < 9; ++k) fc.xyzToRgb[k] = hostColorMatrices().xyzToRec709D65[k];
    return fc;
}

void ptRenderLaunch(const SceneGPU &scene, const PathBuffers &pb, const Film &film, const FrameParams &fpIn,
                    const FilmResolve &resolve, int numSMs, cudaStream_t stream, StageTimer* timer,
                    const GuideFrame* gfp) {
    FrameParams fp = fpIn;
    if (fp.maxPathLength == 0 || fp.maxPathLength > kMaxBounces)
        throw std::runtime_error("maxPathLength out of range");
    StageTimer dummy;
    StageTimer &T = timer ? *timer : dummy;
    // No more blocks than the launch has paths for: late bounces of a small
    // frame would otherwise start thousands of blocks that find no work.
    const int grid = static_cast<int>(std::min<uint32_t>(numSMs * (fp.blocksPerSM ? fp.blocksPerSM : 8),
                                                         (fp.numPaths + 255) / 256));
    const uint32_t rayGrid = std::min<uint32_t>(numSMs * (fp.blocksPerSM ? fp.blocksPerSM : 8) *
                                                    (256 / kRayThreads),
                                                (fp.numPaths + kRayThreads - 1) / kRayThreads);
    const size_t pMain = sizeof(SceneGPU) + sizeof(PathBuffers) + sizeof(FrameParams);
    const Chain chain(stream);
    ck(cudaMemsetAsync(pb.counters, 0, size_t(kMaxBounces + 1) * kCountersPerBounce * 4, stream), "counters");
    const bool guiding = gfp && (gfp->sample || gfp->record);
    if (guiding && gfp->record) {
        T.begin(kStageGuide, stream, sizeof(void*));
        guideCountsKernel<<<1, 1, 0, stream>>>(gfp->counts);
        T.end(stream);
    }
    for (uint32_t b = 0; b < fp.maxPathLength; ++b) {
        fp.bounce = b;
        T.begin(kStageTrace, stream, pMain);
        if (b == 0) launchChained(cameraTraceKernel, rayGrid, kRayThreads, chain, scene, pb, fp);
        else launchChained(traceShadowKernel, rayGrid, kRayThreads, chain, scene, pb, fp);
        T.end(stream);
        if (guiding && gfp->sample && b < gfp->recBounces) {
            GuidedHitSrc src{ scene, pb, fp, gfp->net };
            MixtureDst dst{ src, gfp->lobes, gfp->lobeWeights, gfp->lobeScales };
            auto kern = guide::guideInferKernel<GuidedHitSrc, MixtureDst>;
            ck(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, guide::kInferSmemBytes),
               "infer smem");
            T.begin(kStageGuide, stream, sizeof(guide::Net) + 2 * sizeof(GuidedHitSrc));
            kern<<<numSMs * guide::kInferBlocksPerSM, guide::kInferThreads, guide::kInferSmemBytes, stream>>>(gfp->net, src, dst, gfp->err);
            T.end(stream);
        }
        T.begin(kStageShade, stream, pMain + (guiding ? sizeof(GuideFrame) : 0));
        // the kMaps variants: normal maps, and float3 textures on scalar parameters
        const bool maps = scene.geomMaps != nullptr || scene.hasScalarTextures != 0;
        // the guided variant only where guiding acts: bounces that sample or
        // record, and the one after the last recorded bounce, which closes
        // its records; later bounces only add to the path's contribution,
        // which the plain variant (fewer registers) does the same way
        const bool guideShade = guiding && (b < gfp->recBounces || (gfp->record && b == gfp->recBounces));
        if (guideShade && maps) launchChained(shadeKernel<true, true>, grid, 256, chain, scene, pb, fp, *gfp);
        else if (guideShade) launchChained(shadeKernel<true, false>, grid, 256, chain, scene, pb, fp, *gfp);
        else if (maps) launchChained(shadeKernel<false, true>, grid, 256, chain, scene, pb, fp, GuideFrame{});
        else launchChained(shadeKernel<false, false>, grid, 256, chain, scene, pb, fp, GuideFrame{});
        T.end(stream);
    }
    if (guiding && gfp->record) {
        T.begin(kStageGuide, stream, sizeof(PathBuffers) + sizeof(FrameParams) + sizeof(GuideFrame));
        guideFinalizeKernel<<<grid, 256, 0, stream>>>(pb, fp, *gfp);
        T.end(stream);
    }
    T.begin(kStageFilm, stream, sizeof(PathBuffers) + sizeof(Film) + sizeof(FrameParams) + sizeof(FilmConst) +
                                    sizeof(FilmResolve) + 8);
    const uint32_t pixels = fp.width * fp.height;
    const uint32_t samples = fp.numPaths / pixels;
    const uint32_t lanes = filmLanes(pixels, samples, numSMs);
    const uint32_t filmGrid = static_cast<uint32_t>(
        std::min<uint64_t>((static_cast<uint64_t>(pixels) * lanes + kFilmThreads - 1) / kFilmThreads, numSMs * 24u));
    auto filmPass = [&](auto add) {
        constexpr bool kAdd = decltype(add)::value;
        auto kernel = filmResolveKernel<false, 1, kAdd>;
        if (lanes > 1) kernel = filmResolveKernel<true, 4, kAdd>;
        else if (samples >= 4) kernel = filmResolveKernel<false, 4, kAdd>;
        else if (samples >= 2) kernel = filmResolveKernel<false, 2, kAdd>;
        launchChained(kernel, filmGrid, kFilmThreads, chain, pb, film, fp, filmConst(), resolve, samples, lanes);
    };
    if (resolve.overwrite) filmPass(std::false_type{});
    else filmPass(std::true_type{});
    T.end(stream);
    T.begin(kStageFilm, stream, sizeof(PathBuffers) + 16 + sizeof(FilmResolve));
    launchChained(statsKernel, 1, 32, chain, pb, fp.maxPathLength, film.frames, resolve);
    T.end(stream);
    ck(cudaGetLastError(), "launch");
    T.collect();
}

void launchTraceSorted(const SceneGPU &scene, const PathBuffers &pb, const FrameParams &fp, int grid,
                       cudaStream_t stream) {
    traceKernel<<<grid, 256, 0, stream>>>(scene, pb, fp);
}

void filmClear(const Film &film, cudaStream_t stream) {
    ck(cudaMemsetAsync(film.strata, 0, size_t(film.width) * film.height * kNumStrata * 8, stream), "film clear");
    ck(cudaMemsetAsync(film.frames, 0, 4, stream), "film frames");
}

void filmAddFrames(const Film &film, uint32_t samples, cudaStream_t stream) {
    filmAddFramesKernel<<<1, 1, 0, stream>>>(film.frames, samples);
    ck(cudaGetLastError(), "film frames");
}

void filmToRGBA(const Film &film, float4* out, cudaStream_t stream) {
    const uint32_t n = film.width * film.height;
    filmToRGBAKernel<<<(n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096, 256, 0, stream>>>(film,
                                                                                           filmConst(), out);
    ck(cudaGetLastError(), "film convert");
}

} // namespace vlrb
