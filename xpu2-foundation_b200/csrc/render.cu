// The plain megakernel and the small kernels around it.
//
// An item of a launch is a (chunk, tile position, sample) triple laid out sample-minor, so consecutive items are
// consecutive samples of one pixel: a warp's camera rays are coherent and its film update is one set of FP64 atomics a
// pixel (warp-aggregated atomics) instead of one a sample. The film is the reference's: FP64 sums (rgb + alpha), FP64
// odd-index sums (adaptive frames), U32 counts (async_gpu.cu:320-364).
//
// renderSteps (surface scenes): a bounce at a time, a lane taking the next item as soon as its sample is done, the
// warp's rays walked a node a step by whichever lanes are free (below). renderChunks (volumes, counting launches): persistent warps claim 32
// items at a time (one atomic a warp) and each lane runs its sample's whole path (integrate).
#include "integrator.cuh"
#include "render.h"

namespace x2 {

bool diagnosticKernels() {
#ifdef X2_DIAG
    return true;
#else
    return false;
#endif
}

cudaError_t uploadSobol(const uint32_t directions[17][32]) {
    return cudaMemcpyToSymbol(c_sobol, directions, sizeof(uint32_t) * 17 * 32);
}

namespace {

__device__ __forceinline__ uint32_t tilePixel(uint32_t tile, uint32_t position, uint32_t width, uint32_t height) {
    const uint32_t tilesX = (width + 7) / 8;
    const uint32_t x = (tile % tilesX) * 8 + position % 8;
    const uint32_t y = (tile / tilesX) * 8 + position / 8;
    return x < width && y < height ? y * width + x : ~0u;
}

__device__ __forceinline__ void addCounters(Counters* dst, unsigned long long trace, unsigned long long nee, unsigned long long bsdf,
                                            unsigned long long held, unsigned long long samples, unsigned long long errors) {
    const unsigned full = 0xffffffffu;
#pragma unroll
    for (int off = 16; off; off >>= 1) {
        trace += __shfl_down_sync(full, trace, off);
        nee += __shfl_down_sync(full, nee, off);
        bsdf += __shfl_down_sync(full, bsdf, off);
        held += __shfl_down_sync(full, held, off);
        samples += __shfl_down_sync(full, samples, off);
        errors += __shfl_down_sync(full, errors, off);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&dst->trace, trace);
        atomicAdd(&dst->nee, nee);
        atomicAdd(&dst->bsdf, bsdf);
        atomicAdd(&dst->held, held);
        atomicAdd(&dst->samples, samples);
        atomicAdd(&dst->errors, errors);
    }
}

// Work item `item` of a launch (item < itemCount): its pixel and sample index, or pixel ~0u when it is no sample (past
// its chunk's count, or outside the frame).
__device__ __forceinline__ void itemSample(const RenderArgs& a, unsigned long long item, uint32_t& pixel, uint32_t& index) {
    const unsigned long long perChunk = 64ull * a.samplesPerChunk;
    const unsigned long long chunkIndex = item / perChunk;
    const uint32_t offset = uint32_t(item - chunkIndex * perChunk);
    const uint32_t position = offset / a.samplesPerChunk, s = offset % a.samplesPerChunk;
    const x2_chunk chunk = a.chunks[chunkIndex];
    pixel = ~0u;
    index = 0;
    if (s < chunk.count) {
        pixel = tilePixel(chunk.tile, position, a.scene.config.width, a.scene.config.height);
        index = chunk.first + s;
    }
}

// The film update of a warp step: the lanes that finished a sample of the same pixel are summed by the lowest of them
// (its peers' values added in lane order, whichever lanes they are), which then makes one set of FP64 atomics for the
// pixel. Every lane of the warp calls it; done: the lane finished a sample this step.
__device__ __forceinline__ void warpFilm(const RenderArgs& a, bool done, uint32_t pixel, uint32_t index, float r, float g, float b,
                                         float al) {
    const unsigned full = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t key = done ? pixel : ~0u;
    const uint32_t peers = __match_any_sync(full, key);
    const bool leader = done && lane == uint32_t(__ffs(peers) - 1);
    const bool isOdd = done && (index & 1u) && a.odd;
    const double v0 = done ? double(r) : 0.0, v1 = done ? double(g) : 0.0, v2 = done ? double(b) : 0.0, v3 = done ? double(al) : 0.0;
    double s0 = v0, s1 = v1, s2 = v2, s3 = v3;
    double w0 = isOdd ? v0 : 0.0, w1 = isOdd ? v1 : 0.0, w2 = isOdd ? v2 : 0.0, w3 = isOdd ? v3 : 0.0;
    const double o0 = w0, o1 = w1, o2 = w2, o3 = w3;
    const bool anyOdd = __any_sync(full, isOdd);
    uint32_t rest = leader ? peers & ~(1u << lane) : 0u;
    const uint32_t cnt = leader ? uint32_t(__popc(peers)) : 0u;
    while (__any_sync(full, rest != 0)) {
        const int src = rest ? __ffs(rest) - 1 : int(lane);
        const double t0 = __shfl_sync(full, v0, src), t1 = __shfl_sync(full, v1, src);
        const double t2 = __shfl_sync(full, v2, src), t3 = __shfl_sync(full, v3, src);
        double u0 = 0.0, u1 = 0.0, u2 = 0.0, u3 = 0.0;
        if (anyOdd) {
            u0 = __shfl_sync(full, o0, src);
            u1 = __shfl_sync(full, o1, src);
            u2 = __shfl_sync(full, o2, src);
            u3 = __shfl_sync(full, o3, src);
        }
        if (rest) {
            s0 += t0;
            s1 += t1;
            s2 += t2;
            s3 += t3;
            w0 += u0;
            w1 += u1;
            w2 += u2;
            w3 += u3;
            rest &= rest - 1;
        }
    }
    if (leader) {
        double* s = a.sums + 4ull * key;
        atomicAdd(s, s0);
        atomicAdd(s + 1, s1);
        atomicAdd(s + 2, s2);
        atomicAdd(s + 3, s3);
        atomicAdd(a.counts + key, cnt);
        if (a.odd && (w0 != 0.0 || w1 != 0.0 || w2 != 0.0 || w3 != 0.0)) {
            double* d = a.odd + 4ull * key;
            atomicAdd(d, w0);
            atomicAdd(d + 1, w1);
            atomicAdd(d + 2, w2);
            atomicAdd(d + 3, w3);
        }
    }
}

}  // namespace

template <bool kVolumes, bool kTextures>
__device__ __forceinline__ void renderChunksBody(const RenderArgs& a) {
    const unsigned full = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31u;
    unsigned long long trace = 0, nee = 0, bsdf = 0, held = 0, samples = 0, errors = 0;
    for (;;) {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(a.claimed, 32ull);
        base = __shfl_sync(full, base, 0);
        if (base >= a.itemCount) break;
        const unsigned long long item = base + lane;
        uint32_t pixel = ~0u, index = 0;
        if (item < a.itemCount) itemSample(a, item, pixel, index);
        SampleOut o;
        o.status = X2_SKIP;
        o.rgb[0] = o.rgb[1] = o.rgb[2] = o.alpha = 0.0f;
        if (pixel != ~0u) {
            integrate<kVolumes, kTextures>(a.scene, pixel, index, o);
            trace += o.trace;
            nee += o.nee;
            bsdf += o.bsdf;
            held += o.held;
            if (o.status == X2_DONE) ++samples;
            else if (o.status != X2_SKIP) ++errors;
        }
        warpFilm(a, pixel != ~0u && o.status == X2_DONE, pixel, index, o.rgb[0], o.rgb[1], o.rgb[2], o.alpha);
    }
    addCounters(a.counters, trace, nee, bsdf, held, samples, errors);
}
__global__ void __launch_bounds__(kRenderBlock) renderChunks(RenderArgs a) { renderChunksBody<false, false>(a); }
__global__ void __launch_bounds__(kRenderBlock) renderChunksTextured(RenderArgs a) { renderChunksBody<false, true>(a); }
__global__ void __launch_bounds__(kRenderBlock) renderChunksVolumes(RenderArgs a) { renderChunksBody<true, true>(a); }

// renderSteps: the plain megakernel for surface scenes, a bounce at a time. A lane holds one sample's path (its pending
// rays on a local stack, its radiance) and takes the launch's next item as soon as the sample is done, so a warp never
// waits for its longest path (path regeneration). A warp step is one vertex of every live lane's path: the shadow rays
// its lanes' last vertices made and the closest hits of their next pending rays, walked a node a step by whichever
// lanes are free; then the unoccluded rays' contributions added in their list's order and the next vertices shaded
// (afterTrace, shadeVertex), their shadow rays written to the lanes' lists. That is the order in which integrate (one
// thread a sample, shadow rays traced as they come) adds them, and the steps visit the nodes and test the triangles
// traceClosest / traceAny do, so a sample's radiance is the same bit for bit. Scenes with volumes, vertices with more
// than kStepRecords shadow rays and counting launches use renderChunks.
//
// The walk's rays are the warp's, not their lane's: a vertex makes anything from no shadow ray to one a light, and with
// each lane walking its own list a warp waited for its longest (9.5 of 32 lanes active). So the lists lie in global
// memory (RenderArgs::lists, a warp's own few kilobytes of it, in L1 and L2), the warp's rays are numbered through a
// shared table, closest hits first (their walks are the longest), and a lane whose ray is done takes the next number once
// kStepRefill lanes are free; a ray's outcome goes back to its owner through shared memory. 480x270 at 64 samples over 771k
// triangles: 84.4 ms with lists walked lane by lane, 67.0 so (kStepRefill 2: 69.0, 4: 68.0); the box at 250x190 and 16
// samples 3.05, 2.51.
constexpr uint32_t kStepRefill = 8;
constexpr uint32_t kStepClosest = 31;  // in a ray's number: the owner's pending ray, not a list entry

struct StepSink {
    float4* list;
    uint32_t& n;
    Pending* stack;
    uint32_t& size;
    unsigned long long &nee, &bsdf, &heldRays;
    bool full;  // a shadow ray beyond kStepRecords (the launch checks the scene's bound, so never set)
    __device__ void shadow(const ShadowReq& q, bool fromBsdf) {
        if (fromBsdf) ++bsdf;
        else ++nee;
        if (n < kStepRecords) {
            float4* e = list + 3 * n++;
            e[0] = make_float4(q.origin.x, q.origin.y, q.origin.z, q.near);
            e[1] = make_float4(q.dir.x, q.dir.y, q.dir.z, q.far);
            e[2] = make_float4(q.contribution.x, q.contribution.y, q.contribution.z, 0.0f);
        } else {
            full = true;
        }
    }
    __device__ void held() { ++heldRays; }
    __device__ void vertex(uint32_t, const Bsdf&, V3, const TexHit*) {}
    __device__ uint32_t top(uint32_t) const { return size; }
    __device__ void push(const Pending& p) { stack[size++] = p; }
};

static_assert(kStepRecords < kStepClosest, "a ray's number has five bits for the list entry");
template <bool kTextures>
__device__ __forceinline__ void renderStepsBody(const RenderArgs& a) {
    constexpr uint32_t kWarps = kRenderBlock / 32, kRays = 32 * (kStepRecords + 1);
    __shared__ uint2 shortStacks[kShortStack * kRenderBlock];
    __shared__ uint16_t numbers[kWarps][kRays];   // the warp's rays: owner lane | list entry << 5
    __shared__ uint32_t unoccluded[kWarps][32];   // by owner: its list's unoccluded entries
    __shared__ uint32_t closest[kWarps][32][3];   // by owner: its pending ray's hit (triangle, leaf order, t bits)
    const unsigned full = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const SceneView& s = a.scene;
    const Bvh8 bvh = s.bvh;
    uint32_t* overflow = s.overflow;
    Walk<kShortStack> walk;
    uint2 deep[kStack - kShortStack];
    walk.shortStack = shortStacks + threadIdx.x;
    walk.nodes = walk.tris = 0;
    Pending stack[kMaxPending];
    float4* const lists = a.lists + (size_t(blockIdx.x) * kRenderBlock + 32 * warp) * kStepListWords;  // the warp's
    float4* const list = lists + lane * kStepListWords;
    uint32_t size = 0, n = 0, pixel = 0, index = 0;
    V3 cameraPosition{0, 0, 0}, radiance{0, 0, 0};
    float alpha = 0.0f;
    unsigned long long trace = 0, nee = 0, bsdf = 0, held = 0, samples = 0, errors = 0;
    bool live = false, drained = false;
    for (;;) {
        // Idle lanes take the next items (one atomic a warp); an item that is no sample leaves its lane idle.
        const uint32_t idle = __ballot_sync(full, !live);
        if (idle && !drained) {
            const uint32_t leader = __ffs(idle) - 1, want = __popc(idle);
            unsigned long long base = 0;
            if (lane == leader) base = atomicAdd(a.claimed, (unsigned long long)want);
            base = __shfl_sync(full, base, leader);
            drained = base + want >= a.itemCount;
            if (!live) {
                const unsigned long long item = base + __popc(idle & ((1u << lane) - 1u));
                if (item < a.itemCount) {
                    itemSample(a, item, pixel, index);
                    if (pixel != ~0u) {
                        CameraRay camera;
                        if (cameraRay(s, pixel, index, camera)) {
                            cameraPending(camera, stack[0]);
                            size = 1;
                            n = 0;
                            cameraPosition = camera.origin;
                            radiance = V3{0, 0, 0};
                            alpha = 0.0f;
                            live = true;
                        } else {
                            ++errors;
                        }
                    }
                }
            }
        }
        if (!__any_sync(full, live)) {
            if (drained) break;
            continue;
        }
        // The warp's rays, numbered: the pending rays, then the lists' entries.
        const bool pending = live && size > 0;
        const uint32_t pendings = __ballot_sync(full, pending);
        if (pending) {
            const Pending& next = stack[size - 1];
            list[3 * kStepRecords] = make_float4(next.origin.x, next.origin.y, next.origin.z, next.nearT);
            list[3 * kStepRecords + 1] = make_float4(next.dir.x, next.dir.y, next.dir.z, next.farT);
            numbers[warp][__popc(pendings & ((1u << lane) - 1u))] = uint16_t(lane | (kStepClosest << 5));
        }
        const uint32_t entries = live ? n : 0u;
        uint32_t last = entries;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t v = __shfl_up_sync(full, last, off);
            if (lane >= uint32_t(off)) last += v;
        }
        const uint32_t rays = __popc(pendings) + __shfl_sync(full, last, 31), firstEntry = __popc(pendings) + last - entries;
        for (uint32_t k = 0; k < entries; ++k) numbers[warp][firstEntry + k] = uint16_t(lane | (k << 5));
        unoccluded[warp][lane] = 0;
        __syncwarp();
        uint32_t next = 0, number = 0;
        bool walking = false, any = false;
        RayQ r;
        for (;;) {
            uint32_t lanes = __ballot_sync(full, walking);
            if (next < rays && 32 - __popc(lanes) >= int(kStepRefill)) {
                const uint32_t mine = next + __popc(~lanes & ((1u << lane) - 1u));
                if (!walking && mine < rays) {
                    number = numbers[warp][mine];
                    any = (number >> 5) != kStepClosest;
                    const float4* e = lists + (number & 31u) * kStepListWords + 3 * (any ? number >> 5 : kStepRecords);
                    const float4 r0 = e[0], r1 = e[1];
                    r = makeRay(bvh, r0.x, r0.y, r0.z, r1.x, r1.y, r1.z);
                    if (any) walkStart<true, kShortStack>(walk, r, r0.w, r1.w);
                    else walkStart<false, kShortStack>(walk, r, r0.w, r1.w);
                    walking = true;
                }
                next += 32 - __popc(lanes);
                lanes = __ballot_sync(full, walking);
            }
            if (!lanes) break;
            if (walking && walkStepOverlapKind<kShortStack>(bvh, r, walk, deep, overflow, lanes, any)) {
                const uint32_t owner = number & 31u;
                if (!any) {
                    closest[warp][owner][0] = walk.best;
                    closest[warp][owner][1] = walk.bestLeaf;
                    closest[warp][owner][2] = __float_as_uint(walk.tmax);
                } else if (!walk.best) {
                    atomicOr(&unoccluded[warp][owner], 1u << (number >> 5));
                }
                walking = false;
            }
        }
        __syncwarp();
        // The shadow rays' contributions in the list's order, then the next vertex: the hit rebuilt as trace() does,
        // afterTrace and shadeVertex, its shadow rays to the list.
        for (uint32_t vis = entries ? unoccluded[warp][lane] : 0u; vis; vis &= vis - 1) {
            const float4 c = list[3 * (__ffs(vis) - 1) + 2];
            radiance = add(radiance, V3{c.x, c.y, c.z});
        }
        n = 0;
        if (pending) {
            const uint32_t hitTri = closest[warp][lane][0], hitLeaf = closest[warp][lane][1];
            const float hitT = __uint_as_float(closest[warp][lane][2]);
            Pending pv = stack[--size];
            const uint32_t top = size;
            ++trace;
            Hit hit;
            hit.geom = ~0u;
            hit.prim = 0;
            hit.t = hit.u = hit.v = 0;
            hit.normal = hit.origin = hit.below = hit.point = V3{0, 0, 0};
            V3 va{0, 0, 0}, vb{0, 0, 0}, vc{0, 0, 0};
            if (hitTri != ~0u) {
                const float4* tp = reinterpret_cast<const float4*>(bvh.tris + hitLeaf);
                const float4 A = __ldg(tp), B = __ldg(tp + 1), Cc = __ldg(tp + 2);
                va = V3{A.x, A.y, A.z};
                vb = V3{B.x, B.y, B.z};
                vc = V3{Cc.x, Cc.y, Cc.z};
                hit.geom = __ldg(s.triMesh + hitTri);
                hit.prim = hitTri - __ldg(s.meshFirst + hit.geom);
                hit.t = hitT;
                if (!geometryHit(hit, pv.origin, pv.dir, va, vb, vc)) hit.normal = V3{0, 0, 0};
            }
            const Identity root{pixel, U64(index), U64(s.config.seed), 0};
            afterTrace<false>(s, root, pv, hit, cameraPosition, radiance, alpha);
            if (hit.geom != ~0u) {
                StepSink sink{list, n, stack, size, nee, bsdf, held, false};
                if (!shadeVertex<false, kTextures>(s, root, pixel, index, pv, hit, va, vb, vc, top, radiance, alpha, sink) || sink.full) {
                    ++errors;
                    live = false;
                    n = 0;
                }
            }
        }
        const bool done = live && size == 0 && n == 0;
        if (__any_sync(full, done)) warpFilm(a, done, pixel, index, radiance.x, radiance.y, radiance.z, alpha);
        if (done) {
            ++samples;
            live = false;
        }
    }
    addCounters(a.counters, trace, nee, bsdf, held, samples, errors);
}
template <int kMinBlocks>
__global__ void __launch_bounds__(kRenderBlock, kMinBlocks) renderSteps(RenderArgs a) { renderStepsBody<false>(a); }
template <int kMinBlocks>
__global__ void __launch_bounds__(kRenderBlock, kMinBlocks) renderStepsTextured(RenderArgs a) { renderStepsBody<true>(a); }
template __global__ void renderSteps<4>(RenderArgs);
template __global__ void renderStepsTextured<4>(RenderArgs);

// The per-sample API: integrate() for n (pixel, index) pairs.
template <bool kVolumes, bool kTextures>
__device__ __forceinline__ void integratePairsBody(const SceneView& s, const uint32_t* __restrict__ pairs, unsigned long long n,
                                                   double* __restrict__ rgba, uint32_t* __restrict__ status, Counters* counters) {
    unsigned long long trace = 0, nee = 0, bsdf = 0, held = 0, samples = 0, errors = 0;
    const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
    const unsigned long long first = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
    // Every lane of a warp runs the same number of rounds, so the counters' shuffles below see a full warp.
    const unsigned long long rounds = (n + stride - 1) / stride;
    for (unsigned long long r = 0; r < rounds; ++r) {
        const unsigned long long i = first + r * stride;
        if (i >= n) continue;
        SampleOut o;
        integrate<kVolumes, kTextures>(s, pairs[2 * i], pairs[2 * i + 1], o);
        rgba[4 * i] = double(o.rgb[0]);
        rgba[4 * i + 1] = double(o.rgb[1]);
        rgba[4 * i + 2] = double(o.rgb[2]);
        rgba[4 * i + 3] = double(o.alpha);
        status[i] = o.status;
        trace += o.trace;
        nee += o.nee;
        bsdf += o.bsdf;
        held += o.held;
        if (o.status == X2_DONE) ++samples;
        else errors += o.status == X2_SKIP ? 0 : 1;
    }
    addCounters(counters, trace, nee, bsdf, held, samples, errors);
}
__global__ void __launch_bounds__(kRenderBlock) integratePairs(SceneView s, const uint32_t* __restrict__ pairs, unsigned long long n,
                                                               double* __restrict__ rgba, uint32_t* __restrict__ status, Counters* counters) {
    integratePairsBody<false, false>(s, pairs, n, rgba, status, counters);
}
__global__ void __launch_bounds__(kRenderBlock) integratePairsTextured(SceneView s, const uint32_t* __restrict__ pairs, unsigned long long n,
                                                                       double* __restrict__ rgba, uint32_t* __restrict__ status,
                                                                       Counters* counters) {
    integratePairsBody<false, true>(s, pairs, n, rgba, status, counters);
}
__global__ void __launch_bounds__(kRenderBlock) integratePairsVolumes(SceneView s, const uint32_t* __restrict__ pairs, unsigned long long n,
                                                                      double* __restrict__ rgba, uint32_t* __restrict__ status,
                                                                      Counters* counters) {
    integratePairsBody<true, true>(s, pairs, n, rgba, status, counters);
}

// The ray entry: closest hit and occlusion for n rays (8 floats each: origin, direction, near, far). One thread a ray, both
// walks one after the other: scenes of a few nodes (kRayWalkNodes).
__global__ void traceRaysDirect(SceneView s, const float* __restrict__ rays, unsigned long long n, uint32_t* __restrict__ tri,
                                float* __restrict__ t, uint32_t* __restrict__ occluded) {
    const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
    for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const float* r = rays + 8 * i;
        const RayQ q = makeRay(s.bvh, r[0], r[1], r[2], r[3], r[4], r[5]);
        if (tri || t) {
            float th;
            uint32_t leaf;
            const uint32_t id = traceClosest<false>(s.bvh, q, r[6], r[7], th, &leaf, s.overflow, nullptr);
            if (tri) tri[i] = id;
            if (t) t[i] = id == ~0u ? 0.0f : th;
        }
        if (occluded) occluded[i] = traceAny<false>(s.bvh, q, r[6], r[7], s.overflow, nullptr) ? 1u : 0u;
    }
}

// The same for larger scenes: query 2 i is ray i's closest hit (when a caller wants it), 2 i + 1 its occlusion, walked a node a step by
// persistent warps whose idle lanes take the next queries (as the wavefront's traversal kernels). One thread a ray, both
// walks one after the other, took 0.225 ms for 262,139 scattered rays (0.111 so): a warp waited for its longest walk
// twice. next: the fetch counter, at zero; null where the grid has a lane for every query, which then takes its own (a few
// hundred rays: the counter's clearing alone is a twentieth of the call).
__global__ void __launch_bounds__(kRenderBlock) traceRays(SceneView s, const float* __restrict__ rays, unsigned long long n,
                                                          uint32_t* __restrict__ tri, float* __restrict__ t, uint32_t* __restrict__ occluded,
                                                          unsigned long long* next) {
    __shared__ uint2 shortStacks[kShortStack * kRenderBlock];
    const unsigned full = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31u;
    Walk<kShortStack> walk;
    uint2 deep[kStack - kShortStack];
    walk.shortStack = shortStacks + threadIdx.x;
    walk.nodes = walk.tris = 0;
    const bool wantHit = tri || t, wantOccluded = occluded != nullptr;
    const unsigned long long kinds = (wantHit ? 1u : 0u) + (wantOccluded ? 1u : 0u), queries = n * kinds;
    unsigned long long ray = 0;
    bool walking = false, any = false, drained = queries == 0;
    RayQ r;
    for (;;) {
        uint32_t lanes = __ballot_sync(full, walking);
        if (!drained && 32 - __popc(lanes) >= 8) {
            const uint32_t want = 32 - __popc(lanes);
            unsigned long long base = (unsigned long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31u);
            if (next) {
                if (lane == 0) base = atomicAdd(next, (unsigned long long)want);
                base = __shfl_sync(full, base, 0);
            }
            drained = !next || base + want >= queries;
            const unsigned long long q = base + __popc(~lanes & ((1u << lane) - 1u));
            if (!walking && q < queries) {
                ray = kinds == 2 ? q >> 1 : q;
                any = kinds == 2 ? (q & 1u) != 0 : wantOccluded;
                const float* v = rays + 8 * ray;
                r = makeRay(s.bvh, v[0], v[1], v[2], v[3], v[4], v[5]);
                if (any) walkStart<true, kShortStack>(walk, r, v[6], v[7]);
                else walkStart<false, kShortStack>(walk, r, v[6], v[7]);
                walking = true;
            }
            lanes = __ballot_sync(full, walking);
        }
        if (!lanes) break;
        if (walking && walkStepOverlapKind<kShortStack>(s.bvh, r, walk, deep, s.overflow, lanes, any)) {
            if (any) {
                occluded[ray] = walk.best;
            } else {
                if (tri) tri[ray] = walk.best;
                if (t) t[ray] = walk.best == ~0u ? 0.0f : walk.tmax;
            }
            walking = false;
        }
    }
}

// sample::samplingWord for n identities.
__global__ void sampleWords(const x2_identity* __restrict__ ids, const uint32_t* __restrict__ dims, unsigned long long n, uint32_t policy,
                            uint32_t* __restrict__ out) {
    const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
    for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const x2_identity x = ids[i];
        const Identity id{x.pixel, x.index, x.stream, x.branch};
        const uint32_t d = dims[i];
        if (d >= 16 && d <= 19) {  // the BSDF and light pairs, as the integrator draws them
            uint32_t a, b;
            samplingWordPair(id, d & ~1u, policy, a, b);
            out[i] = d & 1u ? b : a;
        } else {
            out[i] = samplingWord(id, d, policy);
        }
    }
}

// The audit (async_render.h:1010-1040): the first pixel whose count differs from its expected count.
__global__ void auditCounts(const uint32_t* __restrict__ counts, const uint32_t* __restrict__ expected, uint32_t spp, uint32_t pixels,
                            unsigned long long* firstBad) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= pixels) return;
    const uint32_t want = expected ? expected[i] : spp;
    if (counts[i] != want) atomicMin(firstBad, (unsigned long long)i);
}

}  // namespace x2

#ifdef X2_DIAG
// The diagnostic build's switches for this file's kernels (the per-sample API, x2_integrate): mathfn.cuh's mode bits
// and the call record buffer, set on the current device.
extern "C" int x2_diag_set(int mode, void* d_calls, uint32_t capacity) {
    const uint32_t zero = 0;
    x2::mf::DiagCall* calls = static_cast<x2::mf::DiagCall*>(d_calls);
    if (cudaMemcpyToSymbol(x2::mf::g_mode, &mode, sizeof(int)) != cudaSuccess ||
        cudaMemcpyToSymbol(x2::mf::g_calls, &calls, sizeof(calls)) != cudaSuccess ||
        cudaMemcpyToSymbol(x2::mf::g_cap, &capacity, sizeof(uint32_t)) != cudaSuccess ||
        cudaMemcpyToSymbol(x2::mf::g_count, &zero, sizeof(uint32_t)) != cudaSuccess)
        return X2_ECUDA;
    return X2_OK;
}
extern "C" int x2_diag_count(uint32_t* count) {
    return cudaMemcpyFromSymbol(count, x2::mf::g_count, sizeof(uint32_t)) == cudaSuccess ? X2_OK : X2_ECUDA;
}
#endif
