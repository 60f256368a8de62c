// Guide buffers, their linear images and the wavelet denoiser (post.cuh).
#include "post.cuh"
#include "tables.cuh"
#include "wavefront.cuh"

#include <cuda_fp16.h>

#include <algorithm>
#include <stdexcept>

namespace vlrb {
namespace {

size_t align256(size_t b) { return (b + 255) & ~size_t(255); }

void ck(cudaError_t e, const char* what) {
    if (e != cudaSuccess) throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString(e));
}

// getBaseColor of each BSDF (materials.cu:537-539, 592-594, 677-679,
// 805-807, 1077-1081, 1261-1263, 1551-1553, 1702-1704): the albedo or
// coefficient, the conductor's Fresnel reflectance at normal incidence,
// UE4's diffuse + specular F0 colours, zero for emitters.
__device__ __forceinline__ S4 baseColor(const Bsdf &B) {
    switch (B.kind) {
    case kMatte:
    case kLambertianBSDF:
    case kSpecularBRDF:
    case kSpecularBSDF:
    case kMicrofacetBSDF:
        return B.a;
    case kMicrofacetBRDF: {
        FresnelConductor fr{ B.b, B.c };
        return fr.eval(1.0f);
    }
    case kUE4:
        return B.a + B.b;
    default:
        return S4::zero();
    }
}

__device__ __forceinline__ uint64_t mix64(uint64_t z) {
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    return z ^ (z >> 31);
}

// A spectrum tabulated on the 95-sample grid (and its last sample again), at
// one wavelength (blendedEvaluate's interpolation, from shared memory).
__device__ __forceinline__ float tabulatedAt(const float* tab, float lambda) {
    const float p = vclamp<float>((lambda - kWavelengthLow) / (kWavelengthHigh - kWavelengthLow), 0.0f, 1.0f);
    const float binF = p * (kMengSamples - 1);
    const uint32_t bin = vmin<uint32_t>(static_cast<uint32_t>(binF), kMengSamples - 1);
    const float t = binF - bin;
    return tab[bin] * (1 - t) + tab[bin + 1] * t;
}

struct AuxArgs {
    SceneGPU S;
    AuxBuffers ab;
    uint32_t width, height, samples;
    uint64_t seed;
    float white[kMengSamples];   // LightSource Rec.709 (1, 1, 1), the albedo's white point, tabulated
    float xbar[kNumStrata], ybar[kNumStrata], zbar[kNumStrata];
    float xyzToRgb[9];
    double scale;             // 1 / (integral of the CMF x samples so far)
    V3 right, up, forward;    // camera axes (the orientation's matrix columns)
};

// auxBufferGenerator (aux_buffer_generator.cu:21-69): a camera ray per sample
// through the pixel, its first hit's base colour x the white point's
// spectrum / wavelength pdf into the albedo strata, the shading normal
// (normal maps applied) into the normal sum; misses add nothing.  Unlike the
// reference (one hero-wavelength set per sample), each sample evaluates the
// base colour at 16 stratified wavelengths: the denoiser's albedo term needs
// a guide that is smooth after a few samples.  Then copyBuffers
// (post_process.cu:33-91) for the guides: albedo XYZ / samples -> Rec.709;
// the normal sum into the camera frame (inverse orientation), x negated,
// normalised unless zero.
//
// One thread per pixel adds its samples to 16 strata of its own in shared
// memory (odd pitch: no bank conflicts), and the warp moves its 32 pixels'
// strata to the buffer in whole lines: the pixel has one writer, so nothing
// is atomic, and the linear images come from the sums just formed instead of
// a second pass over 128 B a pixel.  kAdd: to what the buffers hold, else in its
// place; its lines are read ahead of the stores (1920 x 1080 guides added: 0.42 ->
// 0.36 ms; the compiler has to keep loads behind stores that it cannot tell apart).
// The white point, the same for every pixel, is tabulated in shared memory;
// upsampling it took six gathers a wavelength (denoised 1080p frame 1.67 -> 1.61
// ms).
constexpr int kAuxThreads = 128, kAuxPitch = kNumStrata + 1;
template <bool kAdd>
__global__ void __launch_bounds__(kAuxThreads) auxKernel(AuxArgs a) {
    __shared__ double sAcc[kAuxThreads * kAuxPitch];
    __shared__ float sWhite[kMengSamples + 1];
    for (uint32_t k = threadIdx.x; k <= kMengSamples; k += kAuxThreads)
        sWhite[k] = a.white[k < kMengSamples ? k : kMengSamples - 1];
    __syncthreads();
    const SceneGPU &S = a.S;
    const Camera &C = S.cam;
    const uint32_t n = a.width * a.height;
    const uint32_t lane = threadIdx.x & 31u;
    double* mine = sAcc + threadIdx.x * kAuxPitch;
    double* warpAcc = sAcc + (threadIdx.x - lane) * kAuxPitch;
    for (uint32_t base = blockIdx.x * kAuxThreads; base < n; base += gridDim.x * kAuxThreads) {
        const uint32_t i = base + threadIdx.x;
        const bool in = i < n;
        const uint32_t px = in ? i % a.width : 0u, py = in ? i / a.width : 0u;
        const uint32_t fi = py * a.ab.stride + px;
#pragma unroll
        for (uint32_t k = 0; k < kNumStrata; ++k) mine[k] = 0.0;
        V3 nsum(0.0f, 0.0f, 0.0f);
        for (uint32_t s = 0; in && s < a.samples; ++s) {
            PCG32 rng{ mix64(a.seed + (static_cast<uint64_t>(i) * a.samples + s) * 0x9E3779B97F4A7C15ULL) };
            const float fx = px + rng.uniform(), fy = py + rng.uniform();
            const float wo = rng.uniform(), ws = rng.uniform();
            float lx, ly;
            const float l0 = rng.uniform(), l1 = rng.uniform();
            concentricDisk(l0, l1, &lx, &ly);
            Frame camFrame;
            camFrame.z = normalize(C.forward);
            camFrame.x = normalize(C.right);
            camFrame.y = cross(camFrame.z, camFrame.x);
            const V3 lensPos = C.right * (C.lensRadius * lx) + C.up * (C.lensRadius * ly) + C.position;
            float dirPDF;
            const V3 dirLocal = cameraSampleDir(C, C.lensRadius * lx, C.lensRadius * ly, fx / a.width,
                                                fy / a.height, &dirPDF);
            const V3 dir = camFrame.fromLocal(dirLocal);
            const Hit h = traceClosest(S, lensPos, dir, FLT_MAX, rng.state);
            if (h.prim == 0xFFFFFFFFu) continue;
            SurfPt sp;
            decodeHit(S, h.prim, h.b1, h.b2, &sp, nullptr);
            const MatDesc &m = S.mats[sp.material];
            const uint32_t parts = m.bsdfKind == kMultiBSDF ? m.numSub : 1u;
            // four wavelength sets at offsets (j + wo) / 4: 16 stratified
            // wavelengths per sample, so the guide is nearly free of
            // spectral noise after a few samples
            for (int j = 0; j < 4; ++j) {
                float selectWLPDF;
                const WLS wls = WLS::equalOffsets((j + wo) * 0.25f, ws, &selectWLPDF);
                // a Multi material's base colour is the sum of its components'
                // (MultiBSDF::getBaseColor, materials.cu:2307-2319)
                S4 base = S4::zero();
                for (uint32_t c = 0; c < parts; ++c) {
                    const MatDesc &mc = m.bsdfKind == kMultiBSDF ? S.mats[m.sub[c]] : m;
                    base += baseColor(buildBsdf(S.meng, mc, wls, sp.tu, sp.tv));
                }
                S4 white;
#pragma unroll
                for (int w = 0; w < 4; ++w) white[w] = tabulatedAt(sWhite, wls.lambda[w]);
                const S4 v = base * white / (4.0f * selectWLPDF);
#pragma unroll
                for (int w = 0; w < 4; ++w) mine[strataBin(wls.lambda[w])] += strataValue(v[w]);
            }
            nsum += sp.frame.z;
        }
        __syncwarp();
        // two pixels' lines per step; what the buffer holds is read ahead of the stores
        auto line = [&](uint32_t r) -> double* {
            const uint32_t j = 2 * r + (lane >> 4);
            const uint32_t fj = __shfl_sync(0xFFFFFFFFu, fi, j);
            return base + (threadIdx.x - lane) + j < n
                       ? a.ab.albedo + static_cast<size_t>(fj) * kNumStrata + (lane & 15u) : nullptr;
        };
        double held[16];
        if (kAdd) {
#pragma unroll
            for (uint32_t r = 0; r < 16; ++r) {
                const double* src = line(r);
                held[r] = src ? *src : 0.0;
            }
        }
#pragma unroll
        for (uint32_t r = 0; r < 16; ++r) {
            double* dst = line(r);
            if (!dst) continue;
            double* sum = warpAcc + (2 * r + (lane >> 4)) * kAuxPitch + (lane & 15u);
            double v = *sum;
            if (kAdd) {
                v += held[r];
                *sum = v;
            }
            *dst = v;
        }
        __syncwarp();
        if (in) {
            if (kAdd) {
                const float4 acc = a.ab.normal[fi];
                nsum = V3(acc.x + nsum.x, acc.y + nsum.y, acc.z + nsum.z);
            }
            a.ab.normal[fi] = make_float4(nsum.x, nsum.y, nsum.z, 0.0f);
            double X = 0, Y = 0, Z = 0;
            for (uint32_t k = 0; k < kNumStrata; ++k) {
                X += a.xbar[k] * mine[k];
                Y += a.ybar[k] * mine[k];
                Z += a.zbar[k] * mine[k];
            }
            const float xyz[3] = { static_cast<float>(X * a.scale), static_cast<float>(Y * a.scale),
                                   static_cast<float>(Z * a.scale) };
            float rgb[3];
            mulColMajor(a.xyzToRgb, xyz, rgb);
            a.ab.linAlbedo[fi] = make_float4(rgb[0], rgb[1], rgb[2], 1.0f);
            const V3 w = nsum;
            V3 c(-dot(w, a.right), dot(w, a.up), dot(w, a.forward));
            if (c.x != 0.0f || c.y != 0.0f || c.z != 0.0f) c = normalize(c);
            a.ab.linNormal[fi] = make_float4(c.x, c.y, c.z, 1.0f);
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------- denoiser
constexpr float kAlbedoEps = 1e-3f;
constexpr float kSigmaLuminance = 4.0f;
// exponent of the normal term: 128 = 2^7 (computed by squaring)
constexpr float kSigmaAlbedo2 = 0.02f;     // 2 x (0.1)^2
constexpr int kWaveletPasses = 5;

struct DenoiseArgs {
    const float4* color;
    const float4* albedo;
    const float4* normal;
    uint4* guide;
    uint32_t width, height, stride;
};

__device__ __forceinline__ uint32_t packHalf2(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    uint32_t u;
    memcpy(&u, &h, 4);
    return u;
}
__device__ __forceinline__ float2 unpackHalf2(uint32_t u) {
    __half2 h;
    memcpy(&h, &u, 4);
    return __half22float2(h);
}

__device__ __forceinline__ bool isGuided(const float4 &a) {
    return a.x + a.y + a.z > kAlbedoEps;
}
__device__ __forceinline__ float luminance(const float4 &c) {
    return 0.2126f * c.x + 0.7152f * c.y + 0.0722f * c.z;
}

// Illumination = colour / albedo (pixels with no albedo, misses and
// emitters, pass through unfiltered), and its luminance variance over the
// 3x3 neighbourhood of guided pixels in .w.
__global__ void demodulateKernel(DenoiseArgs a, float4* illum) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= static_cast<int>(a.width) || y >= static_cast<int>(a.height)) return;
    const size_t p = static_cast<size_t>(y) * a.stride + x;
    const float4 ap = a.albedo[p];
    // the taps' guide record: albedo rgb, normal xyz as halves; albedo r
    // negative marks a pixel that is not filtered
    // (albedo clamped to the largest finite half: an unclamped texture or
    // plug value above it would pack to inf and turn tap weights into NaN)
    const float4 np = a.normal[p];
    constexpr float kHalfMax = 65504.0f;
    a.guide[p] = make_uint4(packHalf2(isGuided(ap) ? fminf(ap.x, kHalfMax) : -1.0f, fminf(ap.y, kHalfMax)),
                            packHalf2(fminf(ap.z, kHalfMax), np.x),
                            packHalf2(np.y, np.z), 0u);
    if (!isGuided(ap)) { illum[p] = make_float4(0.f, 0.f, 0.f, 0.f); return; }
    float sum = 0.0f, sum2 = 0.0f, cnt = 0.0f;
    float4 mine = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int dy = -1; dy <= 1; ++dy)
        for (int dx = -1; dx <= 1; ++dx) {
            const int qx = x + dx, qy = y + dy;
            if (qx < 0 || qy < 0 || qx >= static_cast<int>(a.width) || qy >= static_cast<int>(a.height)) continue;
            const size_t q = static_cast<size_t>(qy) * a.stride + qx;
            const float4 aq = a.albedo[q];
            if (!isGuided(aq)) continue;
            const float4 cq = a.color[q];
            const float4 iq = make_float4(cq.x / fmaxf(aq.x, kAlbedoEps), cq.y / fmaxf(aq.y, kAlbedoEps),
                                          cq.z / fmaxf(aq.z, kAlbedoEps), 0.0f);
            if (dx == 0 && dy == 0) mine = iq;
            const float l = luminance(iq);
            sum += l;
            sum2 += l * l;
            cnt += 1.0f;
        }
    const float mean = sum / cnt;
    mine.w = fmaxf(sum2 / cnt - mean * mean, 0.0f);
    illum[p] = mine;
}

// Two floats per instruction (sm_100a's packed FP32).
struct F2 {
    unsigned long long v;
};
__device__ __forceinline__ F2 f2(float a, float b) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float lo(F2 a) {
    float x, y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
    return x;
}
__device__ __forceinline__ float hi(F2 a) {
    float x, y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
    return y;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}

struct WaveletSums {
    F2 r, g, b, w, v;
};

// The taps q0 and q1 with the same spline weight h around a pixel of albedo
// a*, normal n* and luminance l (all as pairs, a* and l negated).
struct WaveletCentre {
    F2 ax, ay, az, nx, ny, nz, l;
    float recSigmaL;
};
__device__ __forceinline__ void tapPair(const WaveletCentre &c, const uint4 &g0, const uint4 &g1, const float4 &i0,
                                        const float4 &i1, float h0, float h1, WaveletSums &s) {
    const float2 a0 = unpackHalf2(g0.x), b0 = unpackHalf2(g0.y), d0 = unpackHalf2(g0.z);
    const float2 a1 = unpackHalf2(g1.x), b1 = unpackHalf2(g1.y), d1 = unpackHalf2(g1.z);
    if (a0.x < 0.0f) h0 = 0.0f;   // unguided pixels (they hold zeros) have no weight
    if (a1.x < 0.0f) h1 = 0.0f;
    // normal term max(0, n.n')^128 by seven squarings; the albedo and
    // luminance terms in one exponential (one special-function op a tap)
    const F2 dn = fma2(c.nz, f2(d0.y, d1.y), fma2(c.ny, f2(d0.x, d1.x), mul2(c.nx, f2(b0.y, b1.y))));
    F2 wn = f2(fmaxf(0.0f, lo(dn)), fmaxf(0.0f, hi(dn)));
#pragma unroll
    for (int k = 0; k < 7; ++k) wn = mul2(wn, wn);
    const F2 dx = add2(f2(a0.x, a1.x), c.ax), dy = add2(f2(a0.y, a1.y), c.ay), dz = add2(f2(b0.x, b1.x), c.az);
    const F2 da = fma2(dz, dz, fma2(dy, dy, mul2(dx, dx)));
    const F2 r = f2(i0.x, i1.x), g = f2(i0.y, i1.y), b = f2(i0.z, i1.z);
    const F2 dl = fma2(f2(0.0722f, 0.0722f), b, fma2(f2(0.7152f, 0.7152f), g, fma2(f2(0.2126f, 0.2126f), r, c.l)));
    const float e0 = __expf(-lo(da) * (1.0f / kSigmaAlbedo2) - fabsf(lo(dl)) * c.recSigmaL);
    const float e1 = __expf(-hi(da) * (1.0f / kSigmaAlbedo2) - fabsf(hi(dl)) * c.recSigmaL);
    const F2 w = mul2(mul2(f2(h0, h1), wn), f2(e0, e1));
    s.r = fma2(w, r, s.r);
    s.g = fma2(w, g, s.g);
    s.b = fma2(w, b, s.b);
    s.w = add2(s.w, w);
    s.v = fma2(mul2(w, w), f2(i0.w, i1.w), s.v);
}

// One a-trous pass at `step`: 5x5 B3-spline taps at step spacing, each
// weighted by normal agreement, albedo similarity and the luminance
// difference relative to the centre's standard deviation; the variance is
// filtered with the squared weights.  Bound by issue slots (25 taps of about
// 45 instructions): taps that mirror each other share their spline weight, so
// the 24 around the centre run as 12 pairs on packed instructions, and only
// pixels near the border test their taps against the image, in code of their
// own (taps outside it are zeros: weight 0 must not meet an infinite variance).
__global__ void __launch_bounds__(256) waveletKernel(DenoiseArgs a, const float4* in, float4* out, int step) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    const int W = static_cast<int>(a.width), H = static_cast<int>(a.height);
    if (x >= W || y >= H) return;
    const size_t p = static_cast<size_t>(y) * a.stride + x;
    const uint4 gp = a.guide[p];
    const float4 ip = in[p];
    const float2 g0 = unpackHalf2(gp.x), g1 = unpackHalf2(gp.y), g2 = unpackHalf2(gp.z);
    if (g0.x < 0.0f) { out[p] = ip; return; }
    WaveletCentre c;
    c.ax = f2(-g0.x, -g0.x); c.ay = f2(-g0.y, -g0.y); c.az = f2(-g1.x, -g1.x);
    c.nx = f2(g1.y, g1.y); c.ny = f2(g2.x, g2.x); c.nz = f2(g2.y, g2.y);
    const float lp = luminance(ip);
    c.l = f2(-lp, -lp);
    c.recSigmaL = 1.0f / (kSigmaLuminance * sqrtf(ip.w) + 1e-6f);
    constexpr float kSpline[3] = { 3.0f / 8.0f, 1.0f / 4.0f, 1.0f / 16.0f };
    const F2 zero = f2(0.0f, 0.0f);
    WaveletSums s{ zero, zero, zero, zero, zero };
    const int64_t rowStep = static_cast<int64_t>(a.stride) * step;
    auto taps = [&](auto atBorder) {
#pragma unroll
        for (int dy = 0; dy <= 2; ++dy)
#pragma unroll
            for (int dx = dy == 0 ? 1 : -2; dx <= 2; ++dx) {
                // the tap at (dx, dy) and its mirror image
                const float h = kSpline[dx < 0 ? -dx : dx] * kSpline[dy];
                const int64_t off = dy * rowStep + dx * step;
                const int64_t q0 = static_cast<int64_t>(p) + off, q1 = static_cast<int64_t>(p) - off;
                if constexpr (!decltype(atBorder)::value) tapPair(c, a.guide[q0], a.guide[q1], in[q0], in[q1], h, h, s);
                else {
                    const int sx = dx * step, sy = dy * step;
                    const bool in0 = x + sx >= 0 && x + sx < W && y + sy < H;
                    const bool in1 = x - sx >= 0 && x - sx < W && y - sy >= 0;
                    const float4 none = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    tapPair(c, in0 ? a.guide[q0] : gp, in1 ? a.guide[q1] : gp, in0 ? in[q0] : none,
                            in1 ? in[q1] : none, in0 ? h : 0.0f, in1 ? h : 0.0f, s);
                }
            }
    };
    const bool interior = x >= 2 * step && y >= 2 * step && x + 2 * step < W && y + 2 * step < H;
    if (__all_sync(__activemask(), interior)) taps(std::false_type{});
    else taps(std::true_type{});   // the whole warp, so that none runs both
    const float h = kSpline[0] * kSpline[0];
    const float sr = lo(s.r) + hi(s.r) + h * ip.x, sg = lo(s.g) + hi(s.g) + h * ip.y;
    const float sb = lo(s.b) + hi(s.b) + h * ip.z, wsum = lo(s.w) + hi(s.w) + h;
    const float vsum = lo(s.v) + hi(s.v) + h * h * ip.w;
    out[p] = make_float4(sr / wsum, sg / wsum, sb / wsum, vsum / (wsum * wsum));
}

// Colour = filtered illumination x albedo; unguided pixels keep their colour.
__global__ void remodulateKernel(DenoiseArgs a, const float4* illum, float4* color) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= static_cast<int>(a.width) || y >= static_cast<int>(a.height)) return;
    const size_t p = static_cast<size_t>(y) * a.stride + x;
    const float4 ap = a.albedo[p];
    if (!isGuided(ap)) return;
    const float4 ip = illum[p];
    const float w = color[p].w;
    color[p] = make_float4(ip.x * fmaxf(ap.x, kAlbedoEps), ip.y * fmaxf(ap.y, kAlbedoEps),
                           ip.z * fmaxf(ap.z, kAlbedoEps), w);
}

int numSMsOf() {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

} // namespace

size_t auxBufferBytes(uint32_t stride, uint32_t height) {
    const size_t px = static_cast<size_t>(stride) * height;
    return align256(px * kNumStrata * sizeof(double)) + 7 * align256(px * sizeof(float4));
}

void carveAuxBuffers(void* base, uint32_t stride, uint32_t height, AuxBuffers* out) {
    const size_t px = static_cast<size_t>(stride) * height;
    char* c = static_cast<char*>(base);
    out->albedo = reinterpret_cast<double*>(c);
    c += align256(px * kNumStrata * sizeof(double));
    float4** f4[6] = { &out->normal, &out->linAlbedo, &out->linNormal, &out->work[0], &out->work[1], &out->work[2] };
    for (float4** f : f4) {
        *f = reinterpret_cast<float4*>(c);
        c += align256(px * sizeof(float4));
    }
    out->guide = reinterpret_cast<uint4*>(c);
    out->stride = stride;
}

void auxClear(const AuxBuffers &ab, uint32_t height, cudaStream_t stream) {
    const size_t px = static_cast<size_t>(ab.stride) * height;
    ck(cudaMemsetAsync(ab.albedo, 0, px * kNumStrata * sizeof(double), stream), "aux clear");
    ck(cudaMemsetAsync(ab.normal, 0, px * sizeof(float4), stream), "aux clear");
    ck(cudaMemsetAsync(ab.linAlbedo, 0, px * sizeof(float4), stream), "aux clear");
    ck(cudaMemsetAsync(ab.linNormal, 0, px * sizeof(float4), stream), "aux clear");
}

void auxLaunch(const SceneGPU &scene, const AuxBuffers &ab, uint32_t width, uint32_t height, uint32_t samples,
               uint32_t totalSamples, bool overwrite, uint64_t seed, cudaStream_t stream) {
    static const UpSpec white = mengUpsample(hostMengTables(), hostColorMatrices(), SpType::LightSource,
                                             ColorSp::Rec709, 1.0f, 1.0f, 1.0f);
    AuxArgs a;
    mengBlend(hostMengTables(), white, a.white);
    a.S = scene;
    a.ab = ab;
    a.width = width;
    a.height = height;
    a.samples = samples;
    a.seed = seed;
    const CmfStrata &cs = hostCmfStrata();
    for (uint32_t k = 0; k < kNumStrata; ++k) { a.xbar[k] = cs.xbar[k]; a.ybar[k] = cs.ybar[k]; a.zbar[k] = cs.zbar[k]; }
    for (int k = 0; k < 9; ++k) a.xyzToRgb[k] = hostColorMatrices().xyzToRec709D65[k];
    a.scale = 1.0 / (static_cast<double>(cs.integralCMF) * std::max<uint32_t>(totalSamples, 1u));
    a.right = scene.cam.right;
    a.up = scene.cam.up;
    a.forward = scene.cam.forward;
    const uint32_t n = width * height;
    const uint32_t grid = std::min<uint32_t>((n + kAuxThreads - 1) / kAuxThreads,
                                             static_cast<uint32_t>(numSMsOf()) * 16);
    if (grid == 0) return;
    if (overwrite) auxKernel<false><<<grid, kAuxThreads, 0, stream>>>(a);
    else auxKernel<true><<<grid, kAuxThreads, 0, stream>>>(a);
    ck(cudaGetLastError(), "aux kernel");
}

void denoiseLaunch(const AuxBuffers &ab, float4* color, uint32_t width, uint32_t height, cudaStream_t stream) {
    if (width == 0 || height == 0) return;
    DenoiseArgs a{ color, ab.linAlbedo, ab.linNormal, ab.guide, width, height, ab.stride };
    const dim3 block(16, 16), grid((width + 15) / 16, (height + 15) / 16);
    demodulateKernel<<<grid, block, 0, stream>>>(a, ab.work[0]);
    const float4* in = ab.work[0];
    float4* out = ab.work[1];
    for (int pass = 0; pass < kWaveletPasses; ++pass) {
        waveletKernel<<<grid, block, 0, stream>>>(a, in, out, 1 << pass);
        in = out;
        out = out == ab.work[1] ? ab.work[2] : ab.work[1];
    }
    remodulateKernel<<<grid, block, 0, stream>>>(a, in, color);
    ck(cudaGetLastError(), "denoise");
}

} // namespace vlrb
