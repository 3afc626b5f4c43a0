// Kernels of the render path and their arguments (internal to libx2).
#pragma once
#include "integrator.cuh"

namespace x2 {

constexpr int kRenderBlock = 128;
// Shadow rays a vertex may make in the bounce-at-a-time megakernel (light_count x light_samples + bsdf_samples).
constexpr uint32_t kStepRecords = 24;

struct RenderArgs {
    SceneView scene;
    const x2_chunk* chunks;
    unsigned long long itemCount;   // chunks * 64 * samplesPerChunk
    uint32_t samplesPerChunk;
    unsigned long long* claimed;    // the launch's item counter
    double* sums;
    double* odd;                    // null unless the frame is adaptive
    uint32_t* counts;
    Counters* counters;             // the launch's counters
    float4* lists;                  // renderSteps: kStepListWords a thread of the grid
};
// A renderSteps thread's rays in memory the warp's other lanes can walk them from: a vertex's shadow rays (origin and near,
// direction and far, contribution) and the next pending ray (origin and near, direction and far).
constexpr size_t kStepListWords = 3 * size_t(kStepRecords) + 2;

// Whether render.cu is the diagnostic build (its per-sample kernels then record or round as asked).
bool diagnosticKernels();

// Fills the Sobol direction table the render kernels read (this device, current context).
cudaError_t uploadSobol(const uint32_t directions[17][32]);

// The plain megakernel and the per-sample kernel, each in three forms: for scenes without volumes or textures (their
// code compiled out), with textures, and with volumes (and textures).
__global__ void renderChunks(RenderArgs a);
__global__ void renderChunksTextured(RenderArgs a);
__global__ void renderChunksVolumes(RenderArgs a);
// The plain megakernel a bounce at a time (surface scenes whose vertices make at most kStepRecords shadow rays), in
// occupancy variants: kMinBlocks blocks a SM that the register allocation must allow.
template <int kMinBlocks>
__global__ void renderSteps(RenderArgs a);
template <int kMinBlocks>
__global__ void renderStepsTextured(RenderArgs a);
__global__ void integratePairs(SceneView s, const uint32_t* pairs, unsigned long long n, double* rgba, uint32_t* status, Counters* counters);
__global__ void integratePairsTextured(SceneView s, const uint32_t* pairs, unsigned long long n, double* rgba, uint32_t* status,
                                       Counters* counters);
__global__ void integratePairsVolumes(SceneView s, const uint32_t* pairs, unsigned long long n, double* rgba, uint32_t* status,
                                      Counters* counters);
// The ray entry: traceRays for BVHs of at least kRayWalkNodes nodes, traceRaysDirect below, whose few steps are over before
// refilled lanes pay for the fetches. Device us a call for 2,000, 262,139 and a million rays, walked then direct, by the
// BVH's nodes (random triangles, and the closed box): 1 6.3 21.5 59.7, 6.3 16.6 47.3; 2 10.4 41.2 118, 8.4 30.9 97; the box's
// 3 16.6 61.7 177, 12.5 41.2 135; 4 12.5 57.1 160, 12.5 48.4 187; 5 12.4 61.2 178, 12.6 60.4 228; 8 14.8 84.8 265, 20.6 97.7
// 390; 9 18.6 116 379, 20.6 117 533; 14 24.8 150 494, 39.1 194 739. At 4 nodes the direct kernel is the faster for up to some
// hundred thousand rays, from 5 the walked one for all.
constexpr uint32_t kRayWalkNodes = 5;
__global__ void traceRaysDirect(SceneView s, const float* rays, unsigned long long n, uint32_t* tri, float* t, uint32_t* occluded);
__global__ void traceRays(SceneView s, const float* rays, unsigned long long n, uint32_t* tri, float* t, uint32_t* occluded,
                          unsigned long long* next);
__global__ void sampleWords(const x2_identity* ids, const uint32_t* dims, unsigned long long n, uint32_t policy, uint32_t* out);
__global__ void auditCounts(const uint32_t* counts, const uint32_t* expected, uint32_t spp, uint32_t pixels, unsigned long long* firstBad);

}  // namespace x2
