// BSDF shading batch kernel, included by two translation units:
// bsdf_batch.cu compiles it with -fmad=false (every product and sum rounded
// like the reference's host build, for query-by-query parity) and
// bsdf_batch_contracted.cu with FMA contraction on, which is how the
// renderers' kernels compile the same BSDF code.  VLRB_BATCH_NS names the
// namespace of each copy.
//
// Each query = Meng upsampling of the query's RGB albedo and grey IOR,
// construction of one of seven BSDFs, then sample + evaluate + evaluatePDF at
// the sampled direction.
#pragma once

#include "tables.cuh"
#include "vlrb_internal.h"

#include <cuda_runtime.h>

#ifndef VLRB_BATCH_NS
#error "define VLRB_BATCH_NS before including bsdf_batch.cuh"
#endif

namespace vlrb {
namespace VLRB_BATCH_NS {


struct BsdfBatchArgs {
    int64_t n;
    const float* wo;
    const uint32_t* mat;
    const float* rough;
    const float* ior;
    const float* rgb;
    const float* metallic;
    const float* u;
    const float* wl;
    float* value;
    float* pdf;
    float* wi;
    float* evalValue;
    float* evalPdf;
    MengTables tables;
    const ColorMatrices* mats;
    UpSpec oneIOR;   // grey IOR 1 (exterior medium of the dielectric)
    UpSpec zeroIOR;  // zero extinction of the conductors
    int64_t share;   // queries of one group of blocks, a multiple of 8
    int group;       // blocks that work on the same share
};

// Builds the BSDF of material `kind` from the query's immediate parameters in
// the way the reference's setupBSDF callables do (materials.cu:653-661,
// 776-787, 1220-1240, 1516-1536, 1674-1684, 1959-1978).
// K is the BSDF kind (batchKind maps material ids to kinds).
template <uint32_t K>
__device__ __forceinline__ Bsdf buildBatchBsdf(const BsdfBatchArgs &a, int64_t i, const WLS &wls) {
    Bsdf B;
    const ColorMatrices &M = *a.mats;
    const float r = __ldg(a.rgb + 3 * i + 0), g = __ldg(a.rgb + 3 * i + 1), b = __ldg(a.rgb + 3 * i + 2);
    const float eta = __ldg(a.ior + i);
    const float rx = __ldg(a.rough + 2 * i + 0), ry = __ldg(a.rough + 2 * i + 1);
    constexpr uint32_t kind = K;
    B.kind = kind;
    B.flags = 0;
    B.f0 = B.f1 = B.f2 = 0.0f;
    const float alphaX = fmaxf(0.001f, rx * rx);
    const float alphaY = fmaxf(0.001f, ry * ry);
    switch (kind) {
    case kMatte: {
        UpSpec alb = mengUpsample(a.tables, M, SpType::Reflectance, ColorSp::Rec709, r, g, b);
        B.a = mengEvaluate(a.tables, alb, wls);
        break;
    }
    case kSpecularBRDF: {
        UpSpec alb = mengUpsample(a.tables, M, SpType::Reflectance, ColorSp::Rec709, r, g, b);
        UpSpec e = mengUpsample(a.tables, M, SpType::IOR, ColorSp::Rec709, eta, eta, eta);
        B.a = mengEvaluate(a.tables, alb, wls);
        B.b = mengEvaluate(a.tables, e, wls);
        B.c = mengEvaluate(a.tables, a.zeroIOR, wls);
        break;
    }
    case kMicrofacetBRDF: {
        UpSpec e = mengUpsample(a.tables, M, SpType::IOR, ColorSp::Rec709, eta, eta, eta);
        B.b = mengEvaluate(a.tables, e, wls);
        B.c = mengEvaluate(a.tables, a.zeroIOR, wls);
        B.f0 = alphaX; B.f1 = alphaY; B.f2 = 0.0f;
        break;
    }
    case kMicrofacetBSDF: {
        UpSpec alb = mengUpsample(a.tables, M, SpType::Reflectance, ColorSp::Rec709, r, g, b);
        UpSpec e = mengUpsample(a.tables, M, SpType::IOR, ColorSp::Rec709, eta, eta, eta);
        B.a = mengEvaluate(a.tables, alb, wls);
        B.b = mengEvaluate(a.tables, a.oneIOR, wls);
        B.c = mengEvaluate(a.tables, e, wls);
        B.f0 = alphaX; B.f1 = alphaY; B.f2 = 0.0f;
        break;
    }
    case kLambertianBSDF: {
        UpSpec alb = mengUpsample(a.tables, M, SpType::Reflectance, ColorSp::Rec709, r, g, b);
        B.a = mengEvaluate(a.tables, alb, wls);
        B.f0 = 0.04f;
        break;
    }
    case kSpecularBSDF: {
        // SpecularScatteringSurfaceMaterial_setupBSDF (materials.cu:1046-1058):
        // coefficient, exterior IOR 1, interior IOR, dispersive unless a
        // single wavelength is selected
        UpSpec alb = mengUpsample(a.tables, M, SpType::Reflectance, ColorSp::Rec709, r, g, b);
        UpSpec e = mengUpsample(a.tables, M, SpType::IOR, ColorSp::Rec709, eta, eta, eta);
        B.a = mengEvaluate(a.tables, alb, wls);
        B.b = mengEvaluate(a.tables, a.oneIOR, wls);
        B.c = mengEvaluate(a.tables, e, wls);
        B.flags = wls.single ? 0u : 1u;
        break;
    }
    default: {
        UpSpec alb = mengUpsample(a.tables, M, SpType::Reflectance, ColorSp::Rec709, r, g, b);
        S4 base = mengEvaluate(a.tables, alb, wls);
        const float metal = __ldg(a.metallic + i);
        const float specular = 0.5f;
        B.kind = kUE4;
        B.a = base * (1 - metal);
        B.b = lerpS(0.08f * specular * S4::one(), base, metal);
        B.f0 = fmaxf(0.01f, rx);
        break;
    }
    }
    return B;
}

// One query: sample, then evaluate value and pdf at the sampled direction.
template <uint32_t K>
__device__ __forceinline__ void shadeQuery(const BsdfBatchArgs &a, int64_t i) {
    float wlPdf;
    WLS wls = WLS::equalOffsets(__ldg(a.wl + 2 * i + 0), __ldg(a.wl + 2 * i + 1), &wlPdf);
    Bsdf B = buildBatchBsdf<K>(a, i, wls);
    BsdfQuery q;
    q.dirLocal = V3(__ldg(a.wo + 3 * i + 0), __ldg(a.wo + 3 * i + 1), __ldg(a.wo + 3 * i + 2));
    q.wlHint = wls.selected;
    q.filter = dir::All;
    q.importanceMode = 0;
    const float uc = __ldg(a.u + 3 * i + 0), u0 = __ldg(a.u + 3 * i + 1), u1 = __ldg(a.u + 3 * i + 2);
    BsdfSample s;
    s.dirPDF = 0.0f;
    s.dirLocal = V3(0.0f, 0.0f, 0.0f);
    S4 fs = bsdfSampleInternal(B, q, uc, u0, u1, &s, nullptr);
    float4 v4 = make_float4(0.f, 0.f, 0.f, 0.f), e4 = v4;
    float pdf = 0.0f, epdf = 0.0f;
    V3 wi(0.0f, 0.0f, 0.0f);
    if (s.dirPDF > 0.0f) {
        v4 = make_float4(fs[0], fs[1], fs[2], fs[3]);
        pdf = s.dirPDF;
        wi = s.dirLocal;
        S4 ev = bsdfEvalInternal(B, q, wi, nullptr);
        e4 = make_float4(ev[0], ev[1], ev[2], ev[3]);
        epdf = bsdfPDFInternal(B, q, wi, nullptr);
    }
    reinterpret_cast<float4*>(a.value)[i] = v4;
    a.pdf[i] = pdf;
    a.wi[3 * i + 0] = wi.x;
    a.wi[3 * i + 1] = wi.y;
    a.wi[3 * i + 2] = wi.z;
    reinterpret_cast<float4*>(a.evalValue)[i] = e4;
    a.evalPdf[i] = epdf;
}


// Material id -> rank of its BSDF kind in the order the passes run, slowest
// first: ids 0-4 and 6 are their own kinds (6 is SpecularScattering); 5 and
// every id above 6 build the UE4 BSDF, as the reference's default branch does.
__device__ __forceinline__ uint32_t batchRank(uint32_t m) {
    constexpr uint32_t kRankOf = 0x3150246u;   // nibble m: Matte 6, SpecularBRDF 4, GGX 2, GGX BSDF 0, Lambert 5, UE4 1, 6: 3
    return m < 7u ? (kRankOf >> (4 * m)) & 7u : 1u;
}

__device__ __forceinline__ void shadeQueryOfRank(uint32_t rank, const BsdfBatchArgs &a, int64_t i) {
    switch (rank) {
    case 0: shadeQuery<kMicrofacetBSDF>(a, i); break;
    case 1: shadeQuery<kUE4>(a, i); break;
    case 2: shadeQuery<kMicrofacetBRDF>(a, i); break;
    case 3: shadeQuery<kSpecularBSDF>(a, i); break;
    case 4: shadeQuery<kSpecularBRDF>(a, i); break;
    case 5: shadeQuery<kLambertianBSDF>(a, i); break;
    default: shadeQuery<kMatte>(a, i); break;
    }
}

// Queries arrive in random material order.  A block counting-sorts up to
// kTile queries at once by BSDF kind in shared memory (ballots and popcounts,
// three barriers), each kind's run padded to a multiple of 32, and its warps
// take passes of 32 same-kind queries from a shared counter, the slowest kind
// first.  The kernel is bound by latency and instruction fetch inside the GGX
// BSDFs, so what counts is full passes, every warp busy to the end, and the
// warps of a block in the same kind's code at a time: with one list per warp
// (about 300 queries) the last pass of each of the seven kinds left a third
// of the lanes idle, and eight warps ran eight different kinds (2^20 queries:
// 217 -> 185 us).  Inputs are
// gathered from the block's own share (a few KB per array: later kinds find
// the sectors in L2) and outputs go back to the same slots.
//
// A share belongs to a group of blocks: each sorts it, and block g of the
// group takes passes g, g + group, ...  (batchSplit).
constexpr int kBatchThreads = 256;
constexpr int kBatchWarps = kBatchThreads / 32;
constexpr int kTile = 4096;
constexpr int kTilePerLane = kTile / kBatchThreads;
constexpr uint32_t kBatchKinds = 7;
constexpr int kTileSlots = kTile + static_cast<int>(kBatchKinds) * 32;
constexpr uint16_t kBatchPad = 0xFFFFu;

__global__ void __launch_bounds__(kBatchThreads, 3) bsdfBatchKernel(BsdfBatchArgs a) {
    __shared__ uint16_t sIdx[kTileSlots];
    __shared__ uint32_t sCount[kBatchWarps][kBatchKinds + 1];
    __shared__ uint32_t sOff[kBatchKinds + 1];
    __shared__ uint32_t sNext;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t lanesBelow = (1u << lane) - 1u;
    const uint32_t member = blockIdx.x % static_cast<uint32_t>(a.group);
    // shares in multiples of 8 queries: every share starts on a 32-byte
    // sector of every input and output array (4, 8, 12 and 16 B per query)
    const int64_t start = static_cast<int64_t>(blockIdx.x / static_cast<uint32_t>(a.group)) * a.share;
    const int64_t end = start + a.share < a.n ? start + a.share : a.n;
    for (int64_t base = start; base < end; base += kTile) {
        const int count = static_cast<int>(end - base < kTile ? end - base : kTile);
        // the warp's slice of the tile, whole multiples of 32 queries
        const int slice = ((count + kBatchThreads - 1) / kBatchThreads) * 32;
        const int first = static_cast<int>(warp) * slice;
        uint64_t packed = 0;         // ranks of this lane's queries, 3 bits each (7 = none)
        uint32_t counts[kBatchKinds];
#pragma unroll
        for (uint32_t k = 0; k < kBatchKinds; ++k) counts[k] = 0;
#pragma unroll 4
        for (int j = 0; j < kTilePerLane; ++j) {
            if (j * 32 >= slice) break;
            const int li = first + j * 32 + static_cast<int>(lane);
            const uint32_t rank = li < count ? batchRank(__ldg(a.mat + base + li)) : kBatchKinds;
            packed |= static_cast<uint64_t>(rank) << (3 * j);
#pragma unroll
            for (uint32_t k = 0; k < kBatchKinds; ++k) counts[k] += __popc(__ballot_sync(0xFFFFFFFFu, rank == k));
        }
        if (lane == 0) {
#pragma unroll
            for (uint32_t k = 0; k < kBatchKinds; ++k) sCount[warp][k] = counts[k];
        }
        for (int s = static_cast<int>(threadIdx.x); s < kTileSlots; s += kBatchThreads) {
            if (s >= count + static_cast<int>(kBatchKinds) * 32) break;
            sIdx[s] = kBatchPad;
        }
        __syncthreads();
        if (warp == 0) {
            // where each warp's run of each kind begins
            uint32_t total = 0;
            if (lane < kBatchKinds) {
                for (int w = 0; w < kBatchWarps; ++w) {
                    const uint32_t c = sCount[w][lane];
                    sCount[w][lane] = total;
                    total += c;
                }
            }
            const uint32_t padded = (total + 31u) & ~31u;
            uint32_t off = padded;
            for (int o = 1; o < 8; o <<= 1) {
                const uint32_t up = __shfl_up_sync(0xFFFFFFFFu, off, o);
                if (static_cast<int>(lane) >= o) off += up;
            }
            if (lane <= kBatchKinds) sOff[lane] = off - padded;   // lane 7 holds no kind: the end
            if (lane < kBatchKinds)
                for (int w = 0; w < kBatchWarps; ++w) sCount[w][lane] += off - padded;
            if (lane == 0) sNext = 0;
        }
        __syncthreads();
#pragma unroll
        for (uint32_t k = 0; k < kBatchKinds; ++k) counts[k] = sCount[warp][k];
#pragma unroll 4
        for (int j = 0; j < kTilePerLane; ++j) {
            if (j * 32 >= slice) break;
            const uint32_t rank = static_cast<uint32_t>(packed >> (3 * j)) & 7u;
#pragma unroll
            for (uint32_t k = 0; k < kBatchKinds; ++k) {
                const uint32_t bal = __ballot_sync(0xFFFFFFFFu, rank == k);
                if (rank == k) sIdx[counts[k] + __popc(bal & lanesBelow)] = static_cast<uint16_t>(first + j * 32 + lane);
                counts[k] += __popc(bal);
            }
        }
        __syncthreads();
        const uint32_t passes = sOff[kBatchKinds] / 32u;
        for (;;) {
            uint32_t t = 0;
            if (lane == 0) t = atomicAdd(&sNext, 1u);
            t = __shfl_sync(0xFFFFFFFFu, t, 0) * static_cast<uint32_t>(a.group) + member;
            if (t >= passes) break;
            uint32_t rank = 0;
            while (t * 32u >= sOff[rank + 1]) ++rank;
            const uint16_t li = sIdx[t * 32u + lane];
            if (li != kBatchPad) shadeQueryOfRank(rank, a, base + li);
            __syncwarp();
        }
        __syncthreads();
    }
}

// How a batch is split over the grid.  From kAloneShare queries per resident
// block on, each block has a share of its own: it gives every warp about a pass
// and more blocks sort less each.  Below, passes of a few lanes would fill the
// GPU and fetch the same code side by side, so shares of kSmallShare queries,
// whose passes are nearly full, are sorted by several blocks each: with nine
// (half their warps without a pass, the others spread over more SMs) 10,000
// queries took 26.9 us, with the five that give every warp one 29.2.  Queries of seven BSDFs, shares of their own against these: 10,000
// 36.6 and 26.9 us, 20,000 37.1 and 31.5, 40,000 37.3 and 40.8, 100,000 49.6 and 72.3;
// of one (Matte): 20,000 13.3 and 13.3, 100,000 13.2 and 16.7.
constexpr int64_t kAloneShare = 72, kSmallShare = 1024, kSpreadShare = 2048;
struct BatchSplit {
    int64_t share;
    int group, blocks;
};
inline BatchSplit batchSplit(int64_t n, int64_t resident) {
    int64_t share, group = 1;
    if (n >= kAloneShare * resident) {
        share = (n + resident - 1) / resident;
    }
    else {
        share = n < kSmallShare ? n : kSmallShare;
        const int64_t spread = n < kSpreadShare ? n : kSpreadShare;
        group = (spread / 32 + kBatchKinds + kBatchWarps - 1) / kBatchWarps;
    }
    share = (share + 7) & ~int64_t(7);
    const int64_t groups = (n + share - 1) / share;
    return BatchSplit{ share, static_cast<int>(group), static_cast<int>(groups * group) };
}

inline cudaError_t launch(const VLRBBsdfBatch &b, cudaStream_t stream, float* kernelMs) {
    if (b.count <= 0)
        return cudaSuccess;
    static int numSMs = 0, perSM = 0;
    if (numSMs == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&numSMs, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, bsdfBatchKernel, kBatchThreads, 0);
        if (perSM < 1) perSM = 1;
    }
    BsdfBatchArgs a;
    a.n = b.count;
    a.wo = b.wo; a.mat = b.material; a.rough = b.roughness; a.ior = b.ior; a.rgb = b.albedo;
    a.metallic = b.metallic; a.u = b.u; a.wl = b.wavelengthU;
    a.value = b.value; a.pdf = b.pdf; a.wi = b.wi; a.evalValue = b.evalValue; a.evalPdf = b.evalPdf;
    a.tables = deviceMengTables();
    a.mats = deviceColorMatrices();
    const ColorMatrices &hm = hostColorMatrices();
    MengTables ht = hostMengTables();
    a.oneIOR = mengUpsample(ht, hm, SpType::IOR, ColorSp::Rec709, 1.0f, 1.0f, 1.0f);
    a.zeroIOR = mengUpsample(ht, hm, SpType::IOR, ColorSp::Rec709, 0.0f, 0.0f, 0.0f);
    const BatchSplit split = batchSplit(b.count, static_cast<int64_t>(numSMs) * perSM);
    a.share = split.share;
    a.group = split.group;
    const int blocks = split.blocks;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (kernelMs) {
        cudaEventCreate(&e0);
        cudaEventCreate(&e1);
        cudaEventRecord(e0, stream);
    }
    bsdfBatchKernel<<<blocks, kBatchThreads, 0, stream>>>(a);
    cudaError_t err = cudaGetLastError();
    if (kernelMs) {
        cudaEventRecord(e1, stream);
        cudaEventSynchronize(e1);
        cudaEventElapsedTime(kernelMs, e0, e1);
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
    }
    return err;
}

} // namespace VLRB_BATCH_NS
} // namespace vlrb
