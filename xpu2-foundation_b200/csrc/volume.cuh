// Participating media along a path's rays: the reference's volume integration (async_integrator.h:414-591 and
// :616-1291, volume_core.h, volume_grid.h) for VdbVolumes over dense grids, restated for the device with the same
// arithmetic in the same order, so a sample's radiance agrees with the reference's CPU lane.
//
//   crossings     a ray's entries and exits of the volumes' bounds (closed box meshes), found one at a time from
//                 tnear as the reference's backends do (async_cpu.h:1089-1149), then interiority's outermost pairs;
//   march         decoupled ray marching (VolumeMarch::run): each heterogeneous stretch in steps of its least feature
//                 size over the volume quality, the first at a random place in the first step; a step's coefficients
//                 at its end; the transmittance and (camera rays) each volume's emission accumulated; the march stops
//                 below the transmittance threshold;
//   lookups       the light sampling's step lookups re-run the march (ReplaySteps) from the first march's checkpoints
//                 (MarchRecord: every stride steps, the stride doubling as the eight slots fill), the same steps bit
//                 for bit: distance sampling over the steps' weights (pick) and the step at a distance (at);
//   scattering    integrateVolumeScatteringDirect: per light, equi-angular (bounded lights) and distance samples with
//                 MIS, each through the light's source term (a light sample, its surface shadow ray, the volumes'
//                 transmittance on the way by ray marching at the nearest voxel, the Henyey-Greenstein phase);
//   shadows       transmittance(): the volumes' optical thickness along a surface's shadow ray;
//   multiple      (max_volume_depth > 1) the multiple-scattering approximation: scatter events picked from the
//                 march's steps, then free paths from each, each order's extinction, contribution and anisotropy
//                 shrunk by its factor, every light's source term at each event.
//
// Not built: homogeneous BaseVolumes and mapped ones (their ramps and map programs), holdouts (cutouts), motion and
// velocity, emissive regions as light sources, light sets and LPEs; x2_scene_load and x2_config_set refuse scenes and
// configs that would need them.
#pragma once
#include "shading.cuh"

namespace x2 {

constexpr uint32_t kMaxVolumes = 32, kMaxCrossings = 32, kMarchLimit = 1u << 14, kNoGrid = 0xffffffffu;
constexpr uint32_t kDeviceVolumes = 8;  // volumes a scene may hold here (a march keeps an emission sum for each)
constexpr float kVolumeEpsilon = 1.1920928955078125e-07f, kHitEpsilonStart = 1e-5f, kFarLimit = 0.999f * kDistantDistance;
constexpr float kOneOverFourPi = 0.07957747154594766788f;
enum : uint32_t { kOverlapSum = 0, kOverlapMax = 1, kOverlapRnd = 2 };
enum : uint32_t { kEntry = 1, kExit = 2 };
enum : uint32_t { kInterpPoint = 0, kInterpBox = 1, kInterpQuadratic = 2 };

struct Crossing {
    float t;
    uint32_t volume, flags;
};

// ---- component helpers (volume_core.h:197-206) ----
__device__ __forceinline__ V3 vtimes(V3 a, V3 b) { return V3{a.x * b.x, a.y * b.y, a.z * b.z}; }
__device__ __forceinline__ V3 vscaled(V3 a, float s) { return V3{a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ V3 vplus(V3 a, V3 b) { return V3{a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ V3 cmax0(V3 a) { return V3{fmaxf(a.x, 0.0f), fmaxf(a.y, 0.0f), fmaxf(a.z, 0.0f)}; }
// Grey extinction (three equal channels) takes one exponential: equal arguments have equal results.
__device__ __forceinline__ V3 expNeg(V3 a, float s) {
    const float x = mf::exp(-a.x * s);
    if (a.y == a.x && a.z == a.x) return V3{x, x, x};
    return V3{x, mf::exp(-a.y * s), mf::exp(-a.z * s)};
}
__device__ __forceinline__ float vlum(V3 a) { return 0.299f * a.x + 0.587f * a.y + 0.114f * a.z; }
__device__ __forceinline__ bool vblack(V3 a) { return a.x == 0.0f && a.y == 0.0f && a.z == 0.0f; }
__device__ __forceinline__ bool vIsZero(float x) { return fabsf(x) < kVolumeEpsilon; }
__device__ __forceinline__ bool vfinite(float x) { return x - x == 0.0f; }

// ---- dense grids (volume_grid.h:42-134): OpenVDB's world-to-index in doubles, point / box / quadratic sampling ----
// A diagonal map (GridRec::diagonal) leaves out the products with its zeros: they add signed zeros to finite sums.
__device__ __forceinline__ void gridIndex(const GridRec& g, V3 p, double out[3]) {
    const double* m = g.worldToIndex;
    if (g.diagonal) {
        out[0] = double(p.x) * m[0] + m[12];
        out[1] = double(p.y) * m[5] + m[13];
        out[2] = double(p.z) * m[10] + m[14];
        return;
    }
    for (int c = 0; c < 3; ++c) out[c] = double(p.x) * m[0 * 4 + c] + double(p.y) * m[1 * 4 + c] + double(p.z) * m[2 * 4 + c] + m[3 * 4 + c];
}
__device__ __forceinline__ float voxel(const GridRec& g, int i, int j, int k, int c) {
    const int x = i - g.lo[0], y = j - g.lo[1], z = k - g.lo[2];
    if (x < 0 || y < 0 || z < 0 || x >= g.dims[0] || y >= g.dims[1] || z >= g.dims[2]) return 0.0f;
    return __ldg(g.values + g.channels * ((size_t(z) * size_t(g.dims[1]) + size_t(y)) * size_t(g.dims[0]) + size_t(x)) + c);
}
__device__ __forceinline__ float boxLerp(float a, float b, double w) { return a + float(double(b - a) * w); }
__device__ __forceinline__ float quadratic(const float* v, double w) {
    const float a = float(0.5 * double(v[0] + v[2]) - double(v[1])), b = float(0.5 * double(v[2] - v[0])), c = v[1];
    return float(w * (w * double(a) + double(b)) + double(c));
}
// One channel of the grid at p (its world space) by the interpolation mode.
static __device__ __noinline__ float sampleGrid(const GridRec& g, V3 p, uint32_t mode, int c) {
    double ip[3];
    gridIndex(g, p, ip);
    if (mode == kInterpPoint) return voxel(g, int(round(ip[0])), int(round(ip[1])), int(round(ip[2])), c);
    const int i0 = int(floor(ip[0])), j0 = int(floor(ip[1])), k0 = int(floor(ip[2]));
    const double u = ip[0] - i0, v = ip[1] - j0, w = ip[2] - k0;
    if (mode == kInterpBox) {
        float d[2][2][2];
        const int x = i0 - g.lo[0], y = j0 - g.lo[1], z = k0 - g.lo[2];
        if (x >= 0 && y >= 0 && z >= 0 && x < g.dims[0] - 1 && y < g.dims[1] - 1 && z < g.dims[2] - 1) {
            // All eight voxels inside the grid: one base address, no bounds check a voxel.
            const size_t sx = g.channels, sy = sx * size_t(g.dims[0]), sz = sy * size_t(g.dims[1]);
            const float* q = g.values + sz * size_t(z) + sy * size_t(y) + sx * size_t(x) + c;
            for (int i = 0; i < 2; ++i)
                for (int j = 0; j < 2; ++j)
                    for (int k = 0; k < 2; ++k) d[i][j][k] = __ldg(q + i * sx + j * sy + k * sz);
        } else {
            for (int i = 0; i < 2; ++i)
                for (int j = 0; j < 2; ++j)
                    for (int k = 0; k < 2; ++k) d[i][j][k] = voxel(g, i0 + i, j0 + j, k0 + k, c);
        }
        return boxLerp(boxLerp(boxLerp(d[0][0][0], d[0][0][1], w), boxLerp(d[0][1][0], d[0][1][1], w), v),
                       boxLerp(boxLerp(d[1][0][0], d[1][0][1], w), boxLerp(d[1][1][0], d[1][1][1], w), v), u);
    }
    float vx[3];
    for (int i = 0; i < 3; ++i) {
        float vy[3];
        for (int j = 0; j < 3; ++j) {
            const float vz[3] = {voxel(g, i0 - 1 + i, j0 - 1 + j, k0 - 1, c), voxel(g, i0 - 1 + i, j0 - 1 + j, k0, c),
                                 voxel(g, i0 - 1 + i, j0 - 1 + j, k0 + 1, c)};
            vy[j] = quadratic(vz, w);
        }
        vx[i] = quadratic(vy, v);
    }
    return quadratic(vx, u);
}

// ---- a volume's coefficients at a point (localAt, volume_core.h:241-273, for a VdbVolume with no maps) ----
struct VolumeLocal {
    V3 sigmaT, albedo, emission;
    float g;
};
__device__ __forceinline__ V3 affine34(const float* m, V3 p) {
    return V3{m[0] * p.x + m[1] * p.y + m[2] * p.z + m[3], m[4] * p.x + m[5] * p.y + m[6] * p.z + m[7], m[8] * p.x + m[9] * p.y + m[10] * p.z + m[11]};
}
__device__ __forceinline__ V3 gridSpace(const VolumeRec& v, V3 p) {
    if (v.diagonal) return V3{v.worldToGrid[0] * p.x + v.worldToGrid[3], v.worldToGrid[5] * p.y + v.worldToGrid[7], v.worldToGrid[10] * p.z + v.worldToGrid[11]};
    return affine34(v.worldToGrid, p);
}
// A three-channel grid's nearest voxel: one index for the three channels.
static __device__ __noinline__ V3 samplePoint3(const GridRec& g, V3 p) {
    double ip[3];
    gridIndex(g, p, ip);
    const int i = int(round(ip[0])), j = int(round(ip[1])), k = int(round(ip[2]));
    return V3{voxel(g, i, j, k, 0), voxel(g, i, j, k, 1), voxel(g, i, j, k, 2)};
}
// emission: whether the caller reads the emission. Only a camera ray's march does (one step in eleven or so); the replays,
// the shadow marches and the deeper rays leave the emission grid's index and three loads out.
__device__ __forceinline__ VolumeLocal localAt(const SceneView& s, const VolumeRec& v, V3 p, uint32_t interpolation, bool emission) {
    const V3 gp = gridSpace(v, p);
    const float density = v.densityGrid < s.gridCount && s.grids[v.densityGrid].channels == 1 ? sampleGrid(s.grids[v.densityGrid], gp, interpolation, 0) : 0.0f;
    V3 temperature{0, 0, 0};
    if (emission && v.emissionGrid != kNoGrid && v.emissionGrid < s.gridCount && s.grids[v.emissionGrid].channels == 3)
        temperature = samplePoint3(s.grids[v.emissionGrid], gp);
    return VolumeLocal{cmax0(vscaled(v.gain, density)), cmax0(v.colorMult), cmax0(vtimes(temperature, v.incandescence)),
                       fminf(fmaxf(v.g, -1.0f), 1.0f)};
}

// evalShadersAt (volume_core.h:284-378) without holdouts: the regions' volumes combined by the overlap mode.
struct VolumeCoefficients {
    V3 sigmaT, sigmaS;
    float g;
    float surfaceThreshold;
};
static __device__ __noinline__ VolumeCoefficients evalShadersAt(const SceneView& s, uint32_t regions, uint32_t mode, float rnd, V3 p,
                                                         uint32_t interpolationOverride, V3* emissions, uint32_t* chosenVolume) {
    VolumeCoefficients c{{0, 0, 0}, {0, 0, 0}, 0.0f, 1.0f};
    V3 anisotropy{0, 0, 0}, sigmaTSum{0, 0, 0};
    float maxSigmaTLum = -3.402823466e+38f;
    uint32_t first = kMaxVolumes, chosen = kMaxVolumes;
    auto local = [&](uint32_t v) {
        const VolumeRec& vr = s.volumes[v];
        return localAt(s, vr, p, interpolationOverride != kNoGrid ? interpolationOverride : vr.interpolation, emissions != nullptr);
    };
    for (uint32_t v = 0; v < s.config.volume_count; ++v) {
        if (!(regions >> v & 1)) continue;
        const VolumeLocal L = local(v);
        const V3 scatter = vtimes(L.albedo, L.sigmaT);
        if (first == kMaxVolumes) first = v;
        const float l = vlum(L.sigmaT);
        if (mode == kOverlapSum) {
            c.sigmaT = vplus(c.sigmaT, L.sigmaT);
            c.sigmaS = vplus(c.sigmaS, scatter);
            anisotropy = vplus(anisotropy, vscaled(scatter, L.g));
            if (emissions) emissions[v] = L.emission;
            if (l > maxSigmaTLum) {
                maxSigmaTLum = l;
                chosen = v;
            }
        } else if (mode == kOverlapMax) {
            if (l > maxSigmaTLum) {
                maxSigmaTLum = l;
                c.sigmaT = L.sigmaT;
                c.sigmaS = scatter;
                anisotropy = vscaled(scatter, L.g);
                chosen = v;
                if (emissions) emissions[0] = L.emission;
            }
        } else {
            sigmaTSum = vplus(sigmaTSum, L.sigmaT);
        }
    }
    if (mode == kOverlapRnd && first != kMaxVolumes) {
        // The volume rnd picks by its share of the luminance of the summed extinction (each volume's coefficients are
        // evaluated again here: the same values as in the first pass).
        const float total = vlum(sigmaTSum);
        uint32_t pick = first;
        float weight = 1.0f;
        if (total != 0.0f) {
            V3 running{0, 0, 0};
            pick = kMaxVolumes;
            uint32_t last = first;
            for (uint32_t v = 0; v < s.config.volume_count; ++v) {
                if (!(regions >> v & 1)) continue;
                running = vplus(running, local(v).sigmaT);
                last = v;
                if (rnd < vlum(running) / total) {
                    pick = v;
                    break;
                }
            }
            if (pick == kMaxVolumes) pick = last;
            weight = total / vlum(local(pick).sigmaT);
        }
        const VolumeLocal L = local(pick);
        const V3 scatter = vtimes(L.albedo, L.sigmaT);
        c.sigmaT = vscaled(L.sigmaT, weight);
        c.sigmaS = vscaled(scatter, weight);
        anisotropy = vscaled(vscaled(scatter, L.g), weight);
        chosen = pick;
        if (emissions) emissions[0] = vscaled(L.emission, weight);
    }
    if (chosenVolume) *chosenVolume = chosen;
    if (chosen < kMaxVolumes) c.surfaceThreshold = s.volumes[chosen].surfaceThreshold;
    c.g = vlum(anisotropy);
    const float normalization = vlum(c.sigmaS);
    if (normalization > 0.0f) c.g /= normalization;
    return c;
}

// One volume's density lookups along a stretch: what every step reads of its records, in registers. Only for a volume whose
// maps are axis-aligned (VolumeRec::diagonal, GridRec::diagonal) and a density grid of one channel; the lookups give
// sampleGrid's values bit for bit.
struct DensityLookup {
    V3 scale, offset;  // its world to grid space
    double m[3], b[3]; // grid space to index
    const float* values;
    int lo[3], dims[3];
    __device__ V3 gridPoint(V3 p) const { return V3{scale.x * p.x + offset.x, scale.y * p.y + offset.y, scale.z * p.z + offset.z}; }
    __device__ float at(int i, int j, int k) const {
        const int x = i - lo[0], y = j - lo[1], z = k - lo[2];
        if (x < 0 || y < 0 || z < 0 || x >= dims[0] || y >= dims[1] || z >= dims[2]) return 0.0f;
        return __ldg(values + ((size_t(z) * size_t(dims[1]) + size_t(y)) * size_t(dims[0]) + size_t(x)));
    }
    __device__ float box(V3 g) const {
        const double x = double(g.x) * m[0] + b[0], y = double(g.y) * m[1] + b[1], z = double(g.z) * m[2] + b[2];
        const int i = int(floor(x)), j = int(floor(y)), k = int(floor(z));
        const double u = x - i, v = y - j, w = z - k;
        float d[2][2][2];
        const int xx = i - lo[0], yy = j - lo[1], zz = k - lo[2];
        if (xx >= 0 && yy >= 0 && zz >= 0 && xx < dims[0] - 1 && yy < dims[1] - 1 && zz < dims[2] - 1) {
            const size_t sy = size_t(dims[0]), sz = sy * size_t(dims[1]);
            const float* q = values + sz * size_t(zz) + sy * size_t(yy) + size_t(xx);
#pragma unroll
            for (int c = 0; c < 8; ++c) d[c >> 2][(c >> 1) & 1][c & 1] = __ldg(q + (c >> 2) + ((c >> 1) & 1) * sy + (c & 1) * sz);
        } else {
#pragma unroll
            for (int c = 0; c < 8; ++c) d[c >> 2][(c >> 1) & 1][c & 1] = at(i + (c >> 2), j + ((c >> 1) & 1), k + (c & 1));
        }
        return boxLerp(boxLerp(boxLerp(d[0][0][0], d[0][0][1], w), boxLerp(d[0][1][0], d[0][1][1], w), v),
                       boxLerp(boxLerp(d[1][0][0], d[1][0][1], w), boxLerp(d[1][1][0], d[1][1][1], w), v), u);
    }
    __device__ float point(V3 g) const {
        return at(int(round(double(g.x) * m[0] + b[0])), int(round(double(g.y) * m[1] + b[1])), int(round(double(g.z) * m[2] + b[2])));
    }
};
// DensityLookup's nearest voxel with its index made in floats where they decide it: the index's float value is within
// `guard` of the double that sampleGrid rounds (products and sums of values of at most the stretch's ends' size, each
// rounded to 2^-24, under 2^-21 of it together), so unless it lies that close to half way between two voxels both round
// to the same one. Conversions to and from doubles take a quarter of the rate of the rest, six of them a step.
struct NearestVoxel {
    const DensityLookup& d;
    V3 m, b, guard;
    __device__ NearestVoxel(const DensityLookup& lookup, V3 from, V3 to) : d(lookup) {
        const V3 g0 = d.gridPoint(from), g1 = d.gridPoint(to);
        m = V3{float(d.m[0]), float(d.m[1]), float(d.m[2])};
        b = V3{float(d.b[0]), float(d.b[1]), float(d.b[2])};
        auto half = [](float g0, float g1, float m, float b) { return 0.5f - 0x1p-20f * (fmaxf(fabsf(g0), fabsf(g1)) * fabsf(m) + fabsf(b) + 1.0f); };
        guard = V3{half(g0.x, g1.x, m.x, b.x), half(g0.y, g1.y, m.y, b.y), half(g0.z, g1.z, m.z, b.z)};
    }
    // The voxel's value; false where the floats do not decide its index.
    __device__ bool at(V3 p, float& value) const {
        const V3 g = d.gridPoint(p);
        const float magic = 12582912.0f;  // 1.5 x 2^23: adding it rounds to a whole number in the low mantissa bits
        const float x = __fmaf_rn(g.x, m.x, b.x), y = __fmaf_rn(g.y, m.y, b.y), z = __fmaf_rn(g.z, m.z, b.z);
        const float rx = x + magic, ry = y + magic, rz = z + magic;
        const bool sure = fabsf(x - (rx - magic)) < guard.x && fabsf(y - (ry - magic)) < guard.y && fabsf(z - (rz - magic)) < guard.z;
        if (sure) value = d.at(__float_as_int(rx) - 0x4b400000, __float_as_int(ry) - 0x4b400000, __float_as_int(rz) - 0x4b400000);
        return sure;
    }
};
__device__ __forceinline__ bool densityLookup(const SceneView& s, const VolumeRec& v, DensityLookup& d) {
    if (!v.diagonal || v.densityGrid >= s.gridCount) return false;
    const GridRec& g = s.grids[v.densityGrid];
    if (!g.diagonal || g.channels != 1) return false;
    d.scale = V3{v.worldToGrid[0], v.worldToGrid[5], v.worldToGrid[10]};
    d.offset = V3{v.worldToGrid[3], v.worldToGrid[7], v.worldToGrid[11]};
    for (int a = 0; a < 3; ++a) {
        d.m[a] = g.worldToIndex[5 * a];
        d.b[a] = g.worldToIndex[12 + a];
        d.lo[a] = g.lo[a];
        d.dims[a] = g.dims[a];
    }
    d.values = g.values;
    return true;
}

__device__ __forceinline__ float minFeatureSize(const SceneView& s, uint32_t regions) {
    float m = 3.402823466e+38f;
    for (uint32_t v = 0; v < s.config.volume_count; ++v)
        if (regions >> v & 1) m = fminf(m, s.volumes[v].featureSize);
    return m;
}

// ---- crossings (async_cpu.h:1089-1149, with the box meshes' triangles tested one by one) and interiority ----
// The crossings come one at a time, each the nearest triangle past the last one (lowest index first where two are as near);
// a triangle's t does not depend on where the search starts, so every triangle is tested once and the search runs over
// the few that the ray meets (a box: two to four). A ray that meets more than kMet is searched as the backends do,
// triangle by triangle from each crossing.
static __device__ __noinline__ uint32_t volumeCrossings(const SceneView& s, V3 o, V3 d, float tnear, Crossing* x) {
    const RayQ r = makeRay(s.bvh, o.x, o.y, o.z, d.x, d.y, d.z);
    const uint32_t tris = 12u * s.config.volume_count;
    const float inf = __int_as_float(0x7f800000);
    auto test = [&](uint32_t i, float from, float& th) {
        const float* v = s.volumeTris + 9 * i;
        const float4 a = make_float4(v[0], v[1], v[2], 0.0f), b = make_float4(v[3], v[4], v[5], 0.0f), c = make_float4(v[6], v[7], v[8], 0.0f);
        return triTest(r, a, b, c, from, inf, th);
    };
    constexpr uint32_t kMet = 8;
    float metT[kMet];
    uint32_t metTri[kMet];
    uint32_t met = 0;
    for (uint32_t i = 0; i < tris; ++i) {
        float th;
        if (!test(i, tnear, th)) continue;
#pragma unroll
        for (uint32_t m = 0; m < kMet; ++m)
            if (m == met) metT[m] = th, metTri[m] = i;
        ++met;
    }
    uint32_t n = 0;
    float t = tnear;
    for (uint32_t k = 0; k < 4 * kMaxCrossings && n < kMaxCrossings; ++k) {
        float best = inf;
        uint32_t hitTri = ~0u;
        if (met <= kMet) {
#pragma unroll
            for (uint32_t m = 0; m < kMet; ++m)
                if (m < met && metT[m] >= t && metT[m] < best) best = metT[m], hitTri = metTri[m];
        } else {
            for (uint32_t i = 0; i < tris; ++i) {
                float th;
                if (test(i, t, th) && th < best) best = th, hitTri = i;
            }
        }
        if (hitTri == ~0u) break;
        const float* v = s.volumeTris + 9 * hitTri;
        const V3 e1{v[3] - v[0], v[4] - v[1], v[5] - v[2]}, e2{v[6] - v[0], v[7] - v[1], v[8] - v[2]};
        const V3 ng{e1.y * e2.z - e1.z * e2.y, e1.z * e2.x - e1.x * e2.z, e1.x * e2.y - e1.y * e2.x};
        const uint32_t vol = hitTri / 12u;
        const uint32_t flags = d.x * ng.x + d.y * ng.y + d.z * ng.z < 0.0f ? kEntry : kExit;
        if (!(n > 0 && x[n - 1].t == best && x[n - 1].volume == vol && x[n - 1].flags == flags)) x[n++] = Crossing{best, vol, flags};
        t = best + fmaxf(1e-6f, best * 1e-6f);
    }
    return n;
}
// collectVolumeIntervals' interiority (volume_core.h:471-502): only each volume's outermost entry and exit stay; the
// regions the ray starts in are returned.
__device__ __forceinline__ uint32_t interiority(Crossing* x, uint32_t& n) {
    int count[kDeviceVolumes];
    for (uint32_t v = 0; v < kDeviceVolumes; ++v) count[v] = 0;
    uint32_t regions = 0;
    bool redundant = false;
    for (int i = int(n) - 1; i >= 0; --i) {
        const uint32_t v = x[i].volume;
        if (x[i].flags & kEntry) {
            --count[v];
            if (count[v] == 0) regions &= ~(1u << v);
            else if (count[v] > 0) {
                x[i].flags &= ~kEntry;
                redundant = true;
            }
        }
        if (x[i].flags & kExit) {
            if (count[v] == 0) regions |= 1u << v;
            else if (count[v] > 0) {
                x[i].flags &= ~kExit;
                redundant = true;
            }
            ++count[v];
        }
    }
    if (redundant) {
        uint32_t m = 0;
        for (uint32_t i = 0; i < n; ++i)
            if (x[i].flags) x[m++] = x[i];
        n = m;
    }
    return regions;
}
__device__ __forceinline__ void applyCrossing(uint32_t& regions, const Crossing& x) {
    if (x.flags & kEntry) regions |= 1u << x.volume;
    if (x.flags & kExit) regions &= ~(1u << x.volume);
}
__device__ __forceinline__ uint32_t volumeIntervals(const SceneView& s, V3 o, V3 d, float tnear, Crossing* x, uint32_t& regions) {
    uint32_t n = volumeCrossings(s, o, d, tnear, x);
    regions = interiority(x, n);
    return n;
}

// ---- phase function and distance sampling (volume_core.h:505-530) ----
__device__ __forceinline__ float phaseEval(float g, V3 wo, V3 wi) {
    if (fabsf(g) <= 1e-3f) return kOneOverFourPi;
    const float cosTheta = dot(wo, wi), denom = 1 + g * g + 2 * g * cosTheta;
    return vIsZero(denom) ? 0.0f : kOneOverFourPi * (1 - g * g) / (denom * sqrtf(denom));
}
__device__ __forceinline__ float sampleDistanceExponential(float u, float sigma, float a, float b) {
    return a - mf::log(1.0f - u * (1.0f - mf::exp(sigma * (a - b)))) / sigma;
}
__device__ __forceinline__ float pdfDistanceExponential(float t, float sigma, float a, float b) {
    return sigma / (mf::exp((t - a) * sigma) - mf::exp((t - b) * sigma));
}
__device__ __forceinline__ float sampleEquiAngular(float u, float D, float thetaA, float thetaB) { return D * mf::tan((1 - u) * thetaA + u * thetaB); }
__device__ __forceinline__ float pdfEquiAngular(float t, float D, float thetaA, float thetaB) { return D / ((thetaB - thetaA) * (D * D + t * t)); }

// A light's equi-angular pivot (volume_core.h:630-662) for the admitted lights: a point on a rect.
__device__ __forceinline__ bool boundedLight(const x2_light& l) { return l.type != X2_LIGHT_ENV && l.type != X2_LIGHT_DISTANT; }
__device__ __forceinline__ V3 lightPivot(const x2_light& l, const float r[3]) {
    const V3 local{(0.5f - r[0]) * 2.0f * l.half_width, (0.5f - r[1]) * 2.0f * l.half_height, 0.0f};
    return add(V3{l.position[0], l.position[1], l.position[2]}, rowsMul(l.local2render, local));
}

// ---- the march (async_integrator.h:616-798) ----
struct VolumeStep {  // volume::Step without holdouts
    V3 sigmaT, sigmaS, tr;
    float g, tStart, delta;
};
__device__ __forceinline__ float stepWeight(const VolumeStep& s) { return vlum(vtimes(vscaled(s.sigmaS, s.delta), s.tr)) + 0.0f; }

// A place to march again from: 48 bytes, the stream as its next dimension (its words are made again from it).
struct alignas(16) MarchCheckpoint {
    V3 vt;
    float t, stepStart, stepSize, partial;
    uint32_t interval, regions, count, visited, dimension;
};
static_assert(sizeof(MarchCheckpoint) == 48, "three 16-byte words");
// A march's checkpoints, every `stride` steps, the stride doubling once `slots` of them are held.
struct MarchRecord {
    static constexpr uint32_t kSlots = 8;  // of a march inside one thread (in its local memory)
    MarchCheckpoint* at;
    MarchCheckpoint* first = nullptr;  // where the first step is kept (its stepSize 0: not kept), or null
    uint32_t slots;
    uint32_t used = 0, stride = 8, last = 0;
    __device__ MarchRecord(MarchCheckpoint* memory, uint32_t n) : at(memory), slots(n) {}
    __device__ bool wants(uint32_t count) const {
        if (count == 0 || count == last || count % stride) return false;
        return used < slots || count % (2 * stride) == 0;
    }
    __device__ MarchCheckpoint& slot(uint32_t count) {
        if (used == slots) {
            for (uint32_t i = 0; i < slots / 2; ++i) at[i] = at[2 * i + 1];
            used = slots / 2;
            stride *= 2;
        }
        last = count;
        return at[used++];
    }
};

struct VolumeMarch {
    const SceneView& s;
    const Crossing* x;
    uint32_t n, regionsAtStart;
    V3 org, dir;
    float tnear, tfar;
    uint32_t depth;
    bool sampleEmission;
    Stream start;
    uint32_t limit;
    // What a march leaves.
    V3 vt;
    V3 emitted[kDeviceVolumes];
    uint32_t visited, count;
    bool reachedThreshold, stopped;
    MarchRecord* record;
    const float* weightsSoFar;

    template <class Emit>
    __device__ void stepping(Emit& emit, Stream& marching, uint32_t regions, float t1, float t, float stepStart, float stepSize, uint32_t interval) {
        const x2_config& c = s.config;
        // A stretch inside one volume whose lookups DensityLookup makes: evalShadersAt's result for it (sum and max
        // overlap: that volume's own coefficients), with the volume's records read once a stretch, not once a step.
        const bool single = __popc(regions) == 1 && c.volume_overlap_mode != kOverlapRnd;
        const uint32_t only = single ? __ffs(regions) - 1 : 0u;
        const VolumeRec& vr = s.volumes[only];
        DensityLookup density;
        const bool fast = single && vr.interpolation <= kInterpBox && densityLookup(s, vr, density);
        const V3 gain = vr.gain, albedo = cmax0(vr.colorMult);
        const float phase = fminf(fmaxf(vr.g, -1.0f), 1.0f);
        const bool box = vr.interpolation == kInterpBox;
        auto step = [&](float at) {
            V3 emissions[kDeviceVolumes];
            uint32_t chosen = kMaxVolumes;
            VolumeCoefficients k;
            const V3 p = add(org, mul(dir, at));
            if (fast) {
                const V3 gp = density.gridPoint(p);
                k.sigmaT = cmax0(vscaled(gain, box ? density.box(gp) : density.point(gp)));
                k.sigmaS = vtimes(albedo, k.sigmaT);
                k.g = vlum(vscaled(k.sigmaS, phase));
                const float normalization = vlum(k.sigmaS);
                if (normalization > 0.0f) k.g /= normalization;
            } else {
                const float rnd = c.volume_overlap_mode == kOverlapRnd ? marching.next() : 0.0f;
                k = evalShadersAt(s, regions, c.volume_overlap_mode, rnd, p, kNoGrid, sampleEmission ? emissions : nullptr, &chosen);
            }
            const float delta = at - stepStart;
            if (!emit(VolumeStep{k.sigmaT, k.sigmaS, vt, k.g, stepStart, delta}, count)) stopped = true;
            ++count;
            if (fast) {
                if (sampleEmission) {
                    V3 temperature{0, 0, 0};
                    if (vr.emissionGrid != kNoGrid && vr.emissionGrid < s.gridCount && s.grids[vr.emissionGrid].channels == 3)
                        temperature = samplePoint3(s.grids[vr.emissionGrid], density.gridPoint(p));
                    emitted[only] = vplus(emitted[only], vscaled(vtimes(vt, cmax0(vtimes(temperature, vr.incandescence))), delta));
                }
                vt = vtimes(vt, expNeg(k.sigmaT, delta));
                return;
            }
            const V3 te = vt;
            if (sampleEmission) {
                if (c.volume_overlap_mode == kOverlapSum) {
                    for (uint32_t v = 0; v < c.volume_count; ++v)
                        if (regions >> v & 1) emitted[v] = vplus(emitted[v], vscaled(vtimes(te, emissions[v]), delta));
                } else if (chosen < kMaxVolumes) {
                    emitted[chosen] = vplus(emitted[chosen], vscaled(vtimes(te, emissions[0]), delta));
                }
            }
            vt = vtimes(vt, expNeg(k.sigmaT, delta));
        };
        while (t < t1) {
            if (record && count == 0 && record->first)
                *record->first = MarchCheckpoint{vt, t, stepStart, stepSize, 0.0f, interval, regions, 0u, visited, marching.dimension};
            if (record && weightsSoFar && record->wants(count))
                record->slot(count) = MarchCheckpoint{vt, t, stepStart, stepSize, *weightsSoFar, interval, regions, count, visited, marching.dimension};
            if (vlum(vt) < c.volume_transmittance_threshold) {
                reachedThreshold = true;
                return;
            }
            step(t);
            if (stopped) return;
            stepStart = t;
            t += stepSize;
            if (count + 1 >= limit) return;
        }
        if (vlum(vt) < c.volume_transmittance_threshold) {
            reachedThreshold = true;
            return;
        }
        if (t - t1 > kVolumeEpsilon) step(t1);
    }

    template <class Emit>
    __device__ void marchStretch(Emit& emit, Stream& marching, uint32_t regions, float t0, float t1, uint32_t interval) {
        if (!regions || t1 >= kFarLimit || count + 1 >= limit || reachedThreshold || stopped) return;
        visited |= regions;
        // Every admitted volume is heterogeneous: steps of the least feature size over the volume quality (wider
        // deeper in the path), the first at a random place in the first step.
        const float u = marching.next();
        const float stepSize = minFeatureSize(s, regions) * s.config.inv_volume_quality * fmaxf(float(int(depth) - 1), 1.0f);
        stepping(emit, marching, regions, t1, t0 + stepSize * u, t0, stepSize, interval);
    }

    // The march from its start, or from a checkpoint (the same steps from there, bit for bit).
    template <class Emit>
    __device__ void run(Emit& emit, const MarchCheckpoint* from = nullptr) {
        Stream marching = start;
        if (from) {
            marching.dimension = from->dimension;
            marching.group = ~0u;
        }
        uint32_t regions = from ? from->regions : regionsAtStart;
        if (from) {
            vt = from->vt;
            visited = from->visited;
            count = from->count;
        } else {
            vt = V3{1, 1, 1};
            visited = count = 0;
        }
        for (uint32_t v = 0; v < kDeviceVolumes; ++v) emitted[v] = V3{0, 0, 0};
        reachedThreshold = stopped = false;
        float tStart = tnear;
        uint32_t first = 0;
        if (from) {
            const uint32_t k = from->interval;
            stepping(emit, marching, regions, k < n ? x[k].t : tfar, from->t, from->stepStart, from->stepSize, k);
            if (k >= n) return;
            tStart = x[k].t;
            applyCrossing(regions, x[k]);
            first = k + 1;
        }
        for (uint32_t i = first; i < n; ++i) {
            if (x[i].t > tfar || reachedThreshold || stopped) break;
            if (x[i].t - tStart > kVolumeEpsilon) {
                marchStretch(emit, marching, regions, tStart, x[i].t, i);
                tStart = x[i].t;
            }
            applyCrossing(regions, x[i]);
        }
        if (tfar - tStart > kVolumeEpsilon && !reachedThreshold && !stopped) marchStretch(emit, marching, regions, tStart, tfar, n);
    }
};

// The steps as the light sampling asks for them, by marching again (ReplaySteps, async_integrator.h:830-898).
struct ReplaySteps {
    VolumeMarch& m;
    uint32_t count;
    float total;
    bool weightless;
    const MarchRecord* record;
    // The last checkpoint before the march's end for which `before` holds (it holds up to some checkpoint and for none
    // after it: counts, step starts and partial weights only grow), or null.
    template <class Before>
    __device__ const MarchCheckpoint* last(const Before& before) const {
        uint32_t lo = 0, hi = record ? record->used : 0u;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (record->at[mid].count < count && before(record->at[mid])) lo = mid + 1;
            else hi = mid;
        }
        return lo ? &record->at[lo - 1] : nullptr;
    }
    __device__ float cdfBefore(const MarchCheckpoint& c) const { return weightless ? float(c.count) / float(count) : c.partial; }
    __device__ float cdf(float& partial, const VolumeStep& s, uint32_t index) const {
        if (index + 1 >= count) return total;
        if (weightless) return float(index + 1) / float(count);
        partial += stepWeight(s);
        if (partial > total) partial = total;
        return partial;
    }
    // The steps from a checkpoint in registers, while they lie in its stretch and the stretch is in one volume whose lookups
    // DensityLookup makes: VolumeMarch::run keeps the march's state in memory (the replays' callers hold it), a dozen
    // loads and stores a step. False where the stretch ends before emit does (emit's state is then the caller's to
    // reset); a step's g is left to the caller (phaseOf).
    template <class Emit>
    __device__ __forceinline__ bool replay(const MarchCheckpoint* from, Emit& emit) const {
        const SceneView& s = m.s;
        const uint32_t regions = from->regions;
        if (__popc(regions) != 1 || s.config.volume_overlap_mode == kOverlapRnd) return false;
        const VolumeRec& vr = s.volumes[__ffs(regions) - 1];
        DensityLookup density;
        if (vr.interpolation > kInterpBox || !densityLookup(s, vr, density)) return false;
        const V3 gain = vr.gain, albedo = cmax0(vr.colorMult), org = m.org, dir = m.dir;
        const bool box = vr.interpolation == kInterpBox;
        V3 vt = from->vt;
        float t = from->t, stepStart = from->stepStart;
        const float stepSize = from->stepSize, t1 = from->interval < m.n ? m.x[from->interval].t : m.tfar;
        bool inside = true, found = false;
        for (uint32_t i = from->count; inside; ++i) {
            const bool rest = !(t < t1);  // the stretch's last, shorter step
            inside = !rest || t - t1 > kVolumeEpsilon;
            if (inside) {
                const float at = rest ? t1 : t;
                const V3 gp = density.gridPoint(add(org, mul(dir, at)));
                const V3 sigmaT = cmax0(vscaled(gain, box ? density.box(gp) : density.point(gp)));
                const float delta = at - stepStart;
                found = !emit(VolumeStep{sigmaT, vtimes(albedo, sigmaT), vt, 0.0f, stepStart, delta}, i);
                inside = !found && !rest;
                vt = vtimes(vt, expNeg(sigmaT, delta));
                stepStart = t;
                t += stepSize;
            }
        }
        return found;
    }
    __device__ __forceinline__ float phaseOf(const MarchCheckpoint* from, V3 sigmaS) const {
        float g = vlum(vscaled(sigmaS, fminf(fmaxf(m.s.volumes[__ffs(from->regions) - 1].g, -1.0f), 1.0f)));
        const float normalization = vlum(sigmaS);
        if (normalization > 0.0f) g /= normalization;
        return g;
    }
    // Where a replay starts that no checkpoint shortens.
    __device__ __forceinline__ const MarchCheckpoint* start() const {
        return record && record->first && record->first->stepSize > 0.0f ? record->first : nullptr;
    }
    __device__ __noinline__ VolumeStep pick(float r, float& pdf, float& remapped) const {
        const float rw = r * total;
        const MarchCheckpoint* from = last([&](const MarchCheckpoint& c) { return cdfBefore(c) < rw; });
        float partial, prev, found, before;
        VolumeStep chosen{};
        auto reset = [&] { partial = from ? from->partial : 0.0f, prev = from ? cdfBefore(*from) : 0.0f, found = total, before = 0.0f; };
        auto emit = [&](const VolumeStep& s, uint32_t i) {
            const float here = cdf(partial, s, i);
            chosen = s;
            if (here >= rw || i + 1 >= count) {
                found = here, before = prev;
                return false;
            }
            prev = here;
            return true;
        };
        reset();
        const MarchCheckpoint* begin = from ? from : start();
        if (begin && replay(begin, emit)) {
            chosen.g = phaseOf(begin, chosen.sigmaS);
        } else {
            reset();
            m.run(emit, from);
        }
        const float value = found - before;
        pdf = value / total;
        remapped = (rw - before) / value;
        return chosen;
    }
    __device__ __noinline__ VolumeStep at(float t, float& pdf) const {
        const MarchCheckpoint* from = last([&](const MarchCheckpoint& c) { return c.stepStart <= t; });
        float partial, here, kept, keptPrev;
        VolumeStep chosen{};
        auto reset = [&] { partial = from ? from->partial : 0.0f, here = from ? cdfBefore(*from) : 0.0f, kept = 0.0f, keptPrev = 0.0f; };
        auto emit = [&](const VolumeStep& s, uint32_t i) {
            if (i > 0 && s.tStart > t) return false;
            const float before = here;
            here = cdf(partial, s, i);
            chosen = s, kept = here, keptPrev = i > 0 ? before : 0.0f;
            return i + 1 < count;
        };
        reset();
        const MarchCheckpoint* begin = from ? from : start();
        if (begin && replay(begin, emit)) {
            chosen.g = phaseOf(begin, chosen.sigmaS);
        } else {
            reset();
            m.run(emit, from);
        }
        pdf = (kept - keptPrev) / total;
        return chosen;
    }
};

// ---- shadow rays through the volumes (transmittance(), async_integrator.h:425-476) ----
static __device__ __noinline__ V3 volumeTransmittance(const SceneView& s, Stream& st, V3 org, V3 dir, float tnear, float tfar, float scale, int depth) {
    const x2_config& c = s.config;
    Crossing x[kMaxCrossings];
    uint32_t regions;
    const uint32_t n = volumeIntervals(s, org, dir, tnear, x, regions);
    V3 tr{1, 1, 1};
    if (n == 0 && regions == 0) return tr;
    // Loops that leave by their conditions alone (no return or break inside them), so that a warp's lanes meet again at
    // every step whatever each of them found there.
    float tStart = tnear;
    bool through = true, more = true;
    for (uint32_t i = 0; more && through; ++i) {
        more = i < n && x[i].t <= tfar;  // the stretch to crossing i; the last ends at tfar
        const float t0 = tStart, t1 = more ? x[i].t : tfar;
        if (t1 - tStart > kVolumeEpsilon) {
            tStart = t1;
            if (regions && t1 >= kFarLimit) {
                through = false;
            } else if (regions) {
                const float fs = minFeatureSize(s, regions);
                const float tauThreshold = c.volume_transmittance_threshold == 0.0f ? 3.402823466e+38f : -mf::log(c.volume_transmittance_threshold / vlum(tr));
                const float u = st.next();
                const float stepSize = fs * c.inv_volume_shadow_quality * fmaxf(float(depth - 1), 1.0f);
                float t = t0 + stepSize * u;
                V3 tau{0, 0, 0};
                const VolumeRec& vr = s.volumes[__ffs(regions) - 1];
                DensityLookup density;
                if (__popc(regions) == 1 && c.volume_overlap_mode != kOverlapRnd && densityLookup(s, vr, density)) {
                    // One volume, its nearest voxels: four steps' voxels fetched at once, then added and tested in their
                    // order. An index its float does not decide (under one in a hundred) is made in doubles afterwards.
                    const V3 gain = vr.gain;
                    const NearestVoxel nearest(density, add(org, mul(dir, t0)), add(org, mul(dir, t1)));
                    while (t < t1 && through) {
                        float at[4], d[4];
                        uint32_t unsure = 0;
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            at[k] = t;
                            d[k] = 0.0f;
                            if (t < t1 && !nearest.at(add(org, mul(dir, t)), d[k])) unsure |= 1u << k;
                            t += stepSize;
                        }
#pragma unroll 1
                        for (; unsure; unsure &= unsure - 1) {
                            const int k = __ffs(unsure) - 1;
                            const float v = density.point(density.gridPoint(add(org, mul(dir, k == 0 ? at[0] : k == 1 ? at[1] : k == 2 ? at[2] : at[3]))));
#pragma unroll
                            for (int j = 0; j < 4; ++j)
                                if (j == k) d[j] = v;
                        }
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            if (at[k] < t1 && through) {
                                tau = vplus(tau, cmax0(vscaled(gain, d[k])));
                                through = !(vlum(vscaled(tau, stepSize * scale)) > tauThreshold);
                            }
                    }
                } else {
                    while (t < t1 && through) {
                        const float rnd = c.volume_overlap_mode == kOverlapRnd ? st.next() : 0.0f;
                        tau = vplus(tau, evalShadersAt(s, regions, c.volume_overlap_mode, rnd, add(org, mul(dir, t)), kInterpPoint, nullptr, nullptr).sigmaT);
                        through = !(vlum(vscaled(tau, stepSize * scale)) > tauThreshold);
                        t += stepSize;
                    }
                }
                if (through) {
                    tr = vtimes(tr, expNeg(tau, stepSize * scale));
                    through = vlum(tr) > c.volume_transmittance_threshold;
                }
            }
        }
        if (more) applyCrossing(regions, x[i]);
    }
    return through ? tr : V3{0, 0, 0};
}

// estimateInScatteringSourceTermDirect (async_integrator.h:573-591): a light sample from a point in a volume, its
// surface shadow ray, the volumes' transmittance on its way, the phase function.
static __device__ __noinline__ V3 volumeSourceTerm(const SceneView& s, Stream& st, const x2_light& L, V3 P, V3 rayDir, float g, const float ul[3], float scale) {
    V3 wi;
    LightHit lh;
    float r[3] = {ul[0], ul[1], ul[2]};
    if (!lightSample(L, P, nullptr, r, wi, lh)) return V3{0, 0, 0};
    float pdfL;
    const V3 Li = lightEval(L, wi, lh, pdfL);
    if (pdfL == 0.0f || isExactlyZero(Li) || !vfinite(pdfL)) return V3{0, 0, 0};
    float near = kHitEpsilonStart, far = kHitEpsilonEnd * lh.distance;
    near = fmaxf(near, 0.0f);
    far = fmaxf(far - 0.0f, near);
    const float keep = visible(s, P, wi, near, far) ? 1.0f : 0.0f;
    if (keep <= 0.0f) return V3{0, 0, 0};
    const V3 tr = volumeTransmittance(s, st, P, wi, 0.0f, far, scale, 1);
    const float ph = phaseEval(g, V3{-rayDir.x, -rayDir.y, -rayDir.z}, wi);
    return vscaled(vtimes(tr, Li), ph / pdfL * keep);
}

// Henyey-Greenstein sampling about the reversed outgoing direction (volume_core.h phaseSample): uniform over the
// sphere when |g| is at most 1e-3.
__device__ __forceinline__ V3 phaseSample(float g, V3 wo, float u1, float u2) {
    if (fabsf(g) <= 1e-3f) {
        const float cosTheta = 1.0f - 2.0f * u1, sinTheta = sqrtf(fmaxf(0.0f, 1.0f - cosTheta * cosTheta));
        return localSpherical(cosTheta, sinTheta, u2 * kTwoPi);
    }
    u1 = fmaxf(u1, kVolumeEpsilon);
    const float sqrTerm = (1.0f - g * g) / (1.0f - g + 2.0f * g * u1);
    const float cosTheta = (1.0f + g * g - sqrTerm * sqrTerm) / (2.0f * g);
    const float sinTheta = sqrtf(fmaxf(0.0f, 1.0f - cosTheta * cosTheta));
    return localToGlobal(frameN(V3{-wo.x, -wo.y, -wo.z}), localSpherical(cosTheta, sinTheta, kTwoPi * u2));
}

// approximateVolumeMultipleScattering (async_integrator.h:1058-1150, after Wrenninge 2015), pv's volume depth already
// one on: for each of the volume illumination samples, a scatter event picked from the march's steps and a distance
// in it, then free paths from it through the volumes, order after order up to max_volume_depth while the throughput
// stays above the transmittance threshold; at each event every light's source term with the order's attenuation,
// added with the order's contribution factor, and the next direction from the phase function with the order's
// anisotropy. The draws come from one stream a sample, in the reference's order.
static __device__ __noinline__ void volumeMultipleScatter(const SceneView& s, const Identity& root, const Pending& pv, U64 volumeBranch,
                                                          const ReplaySteps& lookup, V3 org, V3 dir, V3 T, V3& radiance) {
    const x2_config& c = s.config;
    if (!(pv.volumeDepth < c.max_volume_depth && c.volume_illumination_samples > 0)) return;
    const uint32_t scatterSamples = c.volume_illumination_samples;
    const float invN = 1.0f / float(scatterSamples);
    for (uint32_t i = 0; i < scatterSamples; ++i) {
        Identity mid = root;
        mid.branch = childBranch(volumeBranch, 0xffff, i);
        Stream ms(mid, pv.depth, 0);
        float pdfDensity, utRemapped;
        const VolumeStep vp = lookup.pick(ms.next(), pdfDensity, utRemapped);
        float sigmaT = vlum(vp.sigmaT);
        const float t0 = vp.tStart, t1 = vp.tStart + vp.delta;
        const float td = sampleDistanceExponential(utRemapped, sigmaT, t0, t1);
        const float pdfT = pdfDensity * pdfDistanceExponential(td, sigmaT, t0, t1);
        if (pdfT == 0.0f || !vfinite(pdfT)) continue;
        const V3 trScatter = vtimes(vp.tr, expNeg(vp.sigmaT, td - t0));
        V3 scatterPoint = add(org, mul(dir, td));
        V3 throughput = vscaled(vtimes(vtimes(T, vp.sigmaS), trScatter), 1.0f / pdfT);
        const float up0 = ms.next(), up1 = ms.next();
        V3 scatterDir = phaseSample(vp.g, V3{-dir.x, -dir.y, -dir.z}, up0, up1);
        for (uint32_t depth = pv.volumeDepth; depth < c.max_volume_depth; ++depth) {
            if (vlum(throughput) < c.volume_transmittance_threshold) break;
            const float ai = mf::pow(c.volume_attenuation_factor, float(depth)), bi = mf::pow(c.volume_contribution_factor, float(depth)),
                        ci = mf::pow(c.volume_phase_attenuation_factor, float(depth));
            const float tFreePath = -mf::log(1.0f - ms.next()) / sigmaT;
            Crossing y[kMaxCrossings];
            uint32_t here;
            const uint32_t m = volumeIntervals(s, scatterPoint, scatterDir, kVolumeEpsilon, y, here);
            for (uint32_t j = 0; j < m && y[j].t <= tFreePath; ++j) applyCrossing(here, y[j]);
            const V3 rayDir = scatterDir;
            scatterPoint = add(scatterPoint, mul(scatterDir, tFreePath));
            if (!here) break;
            const float rnd = c.volume_overlap_mode == kOverlapRnd ? ms.next() : 0.0f;
            const VolumeCoefficients kk = evalShadersAt(s, here, c.volume_overlap_mode, rnd, scatterPoint, kNoGrid, nullptr, nullptr);
            const float g = kk.g * ci;
            sigmaT = vlum(kk.sigmaT);
            if (vIsZero(sigmaT)) break;
            throughput = vscaled(vtimes(throughput, kk.sigmaS), 1.0f / sigmaT);
            for (uint32_t li = 0; li < c.light_count; ++li) {
                const float usl[3] = {ms.next(), ms.next(), ms.next()};
                const V3 Ls = volumeSourceTerm(s, ms, s.lights[li], scatterPoint, rayDir, g, usl, ai);
                radiance = vplus(radiance, vscaled(vtimes(throughput, Ls), invN * bi));
            }
            const float uq0 = ms.next(), uq1 = ms.next();
            scatterDir = phaseSample(g, V3{-rayDir.x, -rayDir.y, -rayDir.z}, uq0, uq1);
        }
    }
}

// One light's scattering sample (integrateVolumeScatteringDirect, async_integrator.h:921-997): its equi-angular part (a
// bounded light's) and its distance part, each zero where the sample has none.
static __device__ __noinline__ void scatterSample(const SceneView& s, const Identity& root, U64 volumeBranch, uint32_t pathDepth,
                                                  const ReplaySteps& lookup, V3 org, V3 dir, V3 T, uint32_t li, uint32_t sample, float firstStart,
                                                  float rayEnd, float invN, V3& equi, V3& distance) {
    const x2_light& L = s.lights[li];
    const bool equiAngular = boundedLight(L);
    equi = distance = V3{0, 0, 0};
    Identity sid = root;
    sid.branch = childBranch(volumeBranch, 1 + li, sample);
    Stream ss(sid, pathDepth, 0);
    float D = 0.0f, thetaA = 0.0f, thetaB = 0.0f, offset = 0.0f;
    float uel[3] = {0.0f, 0.0f, 0.0f};
    if (equiAngular) {
        const float ue = ss.next();
        uel[0] = ss.next();
        uel[1] = ss.next();
        uel[2] = ss.next();
        const V3 pivot = lightPivot(L, uel);
        offset = dot(add(pivot, mul(org, -1.0f)), dir);
        const V3 foot = add(org, mul(dir, offset));
        D = length(add(pivot, mul(foot, -1.0f)));
        thetaA = mf::atan2(firstStart - offset, D);
        thetaB = mf::atan2(rayEnd - offset, D);
        const float te = sampleEquiAngular(ue, D, thetaA, thetaB);
        const float pdfTe = pdfEquiAngular(te, D, thetaA, thetaB);
        if (pdfTe != 0.0f && vfinite(pdfTe)) {
            const float tePrime = te + offset;
            float pdfK;
            const VolumeStep vp = lookup.at(tePrime, pdfK);
            if (!vblack(vp.sigmaS)) {
                const V3 trScatter = vtimes(vp.tr, expNeg(vp.sigmaT, tePrime - vp.tStart));
                float mis = 1.0f;
                const float pdfTd = pdfK * pdfDistanceExponential(tePrime, vlum(vp.sigmaT), vp.tStart, vp.tStart + vp.delta);
                if (vfinite(pdfTd)) mis = powerHeuristic(pdfTe, pdfTd);
                const V3 Ls = volumeSourceTerm(s, ss, L, add(org, mul(dir, tePrime)), dir, vp.g, uel, 1.0f);
                equi = vscaled(vtimes(vtimes(T, vp.sigmaS), vtimes(trScatter, Ls)), invN * mis / pdfTe);
            }
        }
    }
    const float ud = ss.next();
    const float udl[3] = {ss.next(), ss.next(), ss.next()};
    float pdfDensity, udRemapped;
    const VolumeStep vp = lookup.pick(ud, pdfDensity, udRemapped);
    if (pdfDensity == 0.0f) return;
    if (vblack(vp.sigmaS)) return;
    const float sigmaT = vlum(vp.sigmaT), t0 = vp.tStart, t1 = vp.tStart + vp.delta;
    const float td = sampleDistanceExponential(udRemapped, sigmaT, t0, t1);
    const float pdfTd = pdfDensity * pdfDistanceExponential(td, sigmaT, t0, t1);
    if (pdfTd == 0.0f || !vfinite(pdfTd)) return;
    const V3 trScatter = vtimes(vp.tr, expNeg(vp.sigmaT, td - t0));
    float mis = 1.0f;
    if (equiAngular) {
        const float pdfTe = pdfEquiAngular(td - offset, D, thetaA, thetaB);
        if (vfinite(pdfTe)) mis = powerHeuristic(pdfTd, pdfTe);
    }
    // (The diagnostic build's shared-pivot switch gives this sample the equi-angular sample's light
    // point, the pivot its MIS weight was computed with; the reference draws a point of its own.)
    const V3 Ls = volumeSourceTerm(s, ss, L, add(org, mul(dir, td)), dir, vp.g, equiAngular && mf::sharedPivot() ? uel : udl, 1.0f);
    distance = vscaled(vtimes(vtimes(T, vp.sigmaS), vtimes(trScatter, Ls)), invN * mis / pdfTd);
}

// computeRadianceVolume over [tnear, tfar] of a ray (volumeRadiance, async_integrator.h:1152-1291): the camera ray's
// volume emission, the single scattering of every light at the march's steps (a volume depth on), and the path's
// throughput through the volumes. pv's T and volume depth are updated.
static __device__ __noinline__ V3 volumeRadiance(const SceneView& s, const Identity& root, Pending& pv, V3 org, V3 dir, float tnear, float tfar,
                                          V3& alphaTransmittance) {
    const x2_config& c = s.config;
    V3 radiance{0, 0, 0};
    alphaTransmittance = V3{1, 1, 1};
    Crossing x[kMaxCrossings];
    uint32_t regions;
    const uint32_t n = volumeIntervals(s, org, dir, tnear, x, regions);
    if (n == 0 && regions == 0) return radiance;
    const U64 volumeBranch = childBranch(pv.branch, 0xfffc, pv.volumeDepth);
    Identity vid = root;
    vid.branch = childBranch(volumeBranch, 0, 0);
    const bool sampleEmission = pv.depth == 0;
    VolumeMarch march{s, x, n, regions, org, dir, tnear, tfar, pv.depth, sampleEmission, Stream(vid, pv.depth, 0), kMarchLimit};
    float weights = 0.0f, firstStart = 0.0f, lastEnd = 0.0f;
    auto first = [&](const VolumeStep& st, uint32_t i) {
        if (i == 0) firstStart = st.tStart;
        lastEnd = st.tStart + st.delta;
        weights += stepWeight(st);
        return true;
    };
    MarchCheckpoint checkpoints[MarchRecord::kSlots];
    MarchRecord record(checkpoints, MarchRecord::kSlots);
    march.record = &record;
    march.weightsSoFar = &weights;
    march.run(first);
    march.record = nullptr;
    const uint32_t count = march.count;
    if (count == 0) return radiance;
    V3 vt = march.vt, vta = march.vt;
    if (march.reachedThreshold) vt = vta = V3{0, 0, 0};
    alphaTransmittance = vta;
    const V3 T = pv.T;
    if (sampleEmission)
        for (uint32_t v = 0; v < c.volume_count; ++v) {
            if (!(march.visited >> v & 1)) continue;
            const V3 emission = vtimes(T, march.emitted[v]);
            if (vblack(emission)) continue;
            radiance = vplus(radiance, emission);
        }
    if (pv.volumeDepth < c.max_volume_depth) {
        const ReplaySteps lookup{march, count, weights != 0.0f ? weights : 1.0f, weights == 0.0f, &record};
        const float rayEnd = lastEnd;
        // integrateVolumeScatteringDirect (async_integrator.h:921-997).
        const bool highQuality = pv.nonMirror == 0;
        const uint32_t samplesPerLight = highQuality ? c.light_samples : 1, scatterCount = highQuality ? c.volume_illumination_samples : 1;
        if (scatterCount > 0) {
            const float invN = 1.0f / float(samplesPerLight * scatterCount);
            for (uint32_t li = 0; li < c.light_count; ++li) {
                V3 direct{0, 0, 0};
                for (uint32_t k = 0; k < samplesPerLight * scatterCount; ++k) {
                    V3 equi, distance;
                    scatterSample(s, root, volumeBranch, pv.depth, lookup, org, dir, T, li, k, firstStart, rayEnd, invN, equi, distance);
                    direct = vplus(vplus(direct, equi), distance);
                }
                radiance = vplus(radiance, direct);
            }
        }
        ++pv.volumeDepth;
        volumeMultipleScatter(s, root, pv, volumeBranch, lookup, org, dir, T, radiance);
    }
    pv.T = vtimes(pv.T, vt);
    return radiance;
}

// ---- the volumes of a wavefront launch in kernels of their own (wavefront.cu): volumeRadiance in three parts ----
// A ray's volume integral as a launch keeps it a path slot: the first march's result and what its replays need.
struct VolumeHead {
    uint32_t crossings, regions, count, flags;  // kVolumePassed, kVolumeScatters
    float weights, firstStart, lastEnd;
    uint32_t used;                              // checkpoints held
};
enum : uint32_t { kVolumePassed = 1u, kVolumeDeeper = 2u, kVolumeScatters = 4u };

__device__ __forceinline__ VolumeMarch marchOf(const SceneView& s, const Identity& root, const Pending& pv, const Crossing* x, uint32_t n,
                                               uint32_t regions, float tfar, bool emission) {
    Identity vid = root;
    vid.branch = childBranch(childBranch(pv.branch, 0xfffc, pv.volumeDepth), 0, 0);
    return VolumeMarch{s, x, n, regions, pv.origin, pv.dir, pv.nearT, tfar, pv.depth, emission, Stream(vid, pv.depth, 0), kMarchLimit};
}

// The first part of volumeRadiance: the crossings, the march, its transmittance (vt) and a camera ray's emission (added to
// radiance). A march that no scattering sample will replay keeps no weights or checkpoints.
static __device__ __noinline__ void volumeFirstMarch(const SceneView& s, const Identity& root, const Pending& pv, float tfar, Crossing* x,
                                                     MarchCheckpoint* checkpoints, uint32_t slots, VolumeHead& head, V3& vt, V3& radiance) {
    const x2_config& c = s.config;
    head = VolumeHead{0, 0, 0, 0, 0.0f, 0.0f, 0.0f, 0};
    vt = V3{1, 1, 1};
    radiance = V3{0, 0, 0};
    uint32_t regions;
    const uint32_t n = volumeIntervals(s, pv.origin, pv.dir, pv.nearT, x, regions);
    head.crossings = n;
    head.regions = regions;
    if (n == 0 && regions == 0) return;
    const bool sampleEmission = pv.depth == 0, deeper = pv.volumeDepth < c.max_volume_depth;
    const bool scatters = deeper && (pv.nonMirror == 0 ? c.volume_illumination_samples : 1u) > 0;
    VolumeMarch march = marchOf(s, root, pv, x, n, regions, tfar, sampleEmission);
    MarchRecord record(checkpoints, slots - 1);
    record.first = checkpoints + slots - 1;
    if (scatters) record.first->stepSize = 0.0f;
    march.record = scatters ? &record : nullptr;
    float weights = 0.0f, firstStart = 0.0f, lastEnd = 0.0f;
    march.weightsSoFar = &weights;
    if (scatters) {
        auto first = [&](const VolumeStep& st, uint32_t i) {
            if (i == 0) firstStart = st.tStart;
            lastEnd = st.tStart + st.delta;
            weights += stepWeight(st);
            return true;
        };
        march.run(first);
    } else {
        auto pass = [](const VolumeStep&, uint32_t) { return true; };
        march.run(pass);
    }
    head.count = march.count;
    if (march.count == 0) return;
    vt = march.vt;
    if (march.reachedThreshold) vt = V3{0, 0, 0};
    if (sampleEmission)
        for (uint32_t v = 0; v < c.volume_count; ++v) {
            if (!(march.visited >> v & 1)) continue;
            const V3 emission = vtimes(pv.T, march.emitted[v]);
            if (vblack(emission)) continue;
            radiance = vplus(radiance, emission);
        }
    head.flags = kVolumePassed | (deeper ? kVolumeDeeper : 0u) | (scatters ? kVolumeScatters : 0u);
    head.weights = weights;
    head.firstStart = firstStart;
    head.lastEnd = lastEnd;
    head.used = record.used;
}

// The second: sample k of every light's scattering samples (light k / samples, its sample k % samples).
__device__ __forceinline__ void volumeScatterTask(const SceneView& s, const Identity& root, const Pending& pv, float tfar, const Crossing* x,
                                                  MarchCheckpoint* checkpoints, uint32_t slots, const VolumeHead& head, uint32_t k, V3& equi,
                                                  V3& distance) {
    const x2_config& c = s.config;
    const bool highQuality = pv.nonMirror == 0;
    const uint32_t samples = highQuality ? c.light_samples * c.volume_illumination_samples : 1u;
    VolumeMarch march = marchOf(s, root, pv, x, head.crossings, head.regions, tfar, false);
    march.record = nullptr;
    march.weightsSoFar = nullptr;
    MarchRecord record(checkpoints, slots - 1);
    record.first = checkpoints + slots - 1;
    record.used = head.used;
    const ReplaySteps lookup{march, head.count, head.weights != 0.0f ? head.weights : 1.0f, head.weights == 0.0f, &record};
    scatterSample(s, root, childBranch(pv.branch, 0xfffc, pv.volumeDepth), pv.depth, lookup, pv.origin, pv.dir, pv.T, k / samples, k % samples,
                  head.firstStart, head.lastEnd, 1.0f / float(samples), equi, distance);
}

}  // namespace x2
