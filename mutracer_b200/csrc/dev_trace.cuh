// Device sampler (Owen-scrambled Sobol, ZSobol, PCG4D) and two-level BVH2
// traversal with the watertight FP32 triangle test.
#pragma once
#include "../../include/mutracer_b200.h"
#include "dev_math.cuh"

namespace mt {

// Device copy of the bind groups; all pointers are device pointers.
struct DevScene {
  const float4 *bvh;
  const float4 *ins;
  const uint32_t *attr;
  const float4 *mats;
  const float4 *env;
  const float2 *envDist;
  const float4 *lightData;
  const float *lut;
  const float4 *lights;
  uint32_t envW, envH;
  uint32_t vstride, vnormalOff, vnormalFloat;
  uint32_t flags;
  uint32_t insCount, matCount;
  const float4 *maps;       // MTC_MAP_VEC4_ROWS per material map
  const float4 *mapTexels;  // RGBA per texel
  uint32_t mapCount, mapTexelCount;
  uint32_t vuvOff;          // word offset of the f32 UV pair (0: no UVs)
  uint32_t vcolorOff, vcolorFloat;  // vertex color word(s) (0: white), f32x3 or RGBA8
  uint32_t vuv1Off;         // secondary UV pair (0: the primary pair)
  const uint32_t *triMats;  // material + 1 per bvh vec4 (null: instance materials only)
};

// One render job: scene, uniforms, outputs (the plain kernel takes one as a
// __grid_constant__ parameter; the batched kernel reads a table of them).
struct JobData {
  DevScene s;
  mtc_trace_uniform u;
  mtc_camera_uniform cam;
  float4 *outColor, *outNormal, *outAlbedo, *outCatcher;
  uint32_t samples;
  uint32_t width, height;
  uint32_t tilesX, tilesY;
  uint32_t firstItem;  // first global work item of this job (batched kernel)
  uint32_t items;      // tiles * samples
  uint32_t _pad;
};

struct Counters {
  uint32_t ext = 0, shadow = 0;
};

// ------------------------------------------------------------------ sampler
// sobol.wgsl.ts:23-45
MTD uint32_t sampleHash(uint32_t x) {
  x ^= x >> 16; x *= 0x7feb352du;
  x ^= x >> 15; x *= 0x846ca68bu;
  return x ^ (x >> 16);
}
MTD uint32_t sampleSeed(uint32_t a, uint32_t b) { return sampleHash(a ^ sampleHash(b + 0x9e3779b9u)); }
MTD uint32_t lkPermute(uint32_t v, uint32_t seed) {
  uint32_t x = v + seed;
  x ^= x * 0x6c50b47cu; x ^= x * 0xb82f1e52u;
  x ^= x * 0xc7afe638u; x ^= x * 0x8d22f6e6u;
  return x;
}
MTD uint32_t owen(uint32_t x, uint32_t seed) { return __brev(lkPermute(__brev(x), seed)); }
MTD uint32_t sobolD1(uint32_t v) {
  uint32_t r = __brev(v);
  r ^= (r << 1) & 0xaaaaaaaau;
  r ^= (r << 2) & 0xccccccccu;
  r ^= (r << 4) & 0xf0f0f0f0u;
  r ^= (r << 8) & 0xff00ff00u;
  r ^= (r << 16) & 0xffff0000u;
  return r;
}
MTD uint32_t morton2(uint32_t x, uint32_t y) {
  uint32_t vx = x & 255u, vy = y & 255u;
  vx = (vx | (vx << 4)) & 0x0f0fu; vy = (vy | (vy << 4)) & 0x0f0fu;
  vx = (vx | (vx << 2)) & 0x3333u; vy = (vy | (vy << 2)) & 0x3333u;
  vx = (vx | (vx << 1)) & 0x5555u; vy = (vy | (vy << 1)) & 0x5555u;
  return vx | (vy << 1);
}
// Packed pbrt-v4 ZSobol digit permutations (src/renderer/sampling.ts:23-28).
__device__ __constant__ static const uint32_t kZPermWords[6] = {
    0x78d8b4e4u, 0xb1e19c6cu, 0x8d2d39c9u, 0x72d236c6u, 0x87271e4eu, 0x93634b1bu};
MTD uint32_t zSobolPermutation(uint32_t perm) {
  return (kZPermWords[perm >> 2] >> ((perm & 3u) * 8u)) & 255u;
}
MTD uint32_t zSobolIndex(uint32_t morton, uint32_t dim, uint32_t logSPP) {
  uint32_t odd = logSPP & 1u;
  uint32_t digits = 8u + ((logSPP + 1u) >> 1);
  uint32_t result = 0;
  for (int digit = int(digits) - 1; digit >= int(odd); digit--) {
    uint32_t shift = 2u * uint32_t(digit) - odd;
    uint32_t higher = shift < 30u ? morton >> (shift + 2u) : 0u;
    uint32_t perm = (sampleHash(higher ^ (0x55555555u * dim)) >> 24) % 24u;
    uint32_t d = (morton >> shift) & 3u;
    result |= ((zSobolPermutation(perm) >> (2u * d)) & 3u) << shift;
  }
  if (odd != 0u) result |= (morton & 1u) ^ (sampleHash((morton >> 1) ^ (0x55555555u * dim)) & 1u);
  return result;
}

struct Sampler {
  uint32_t px, py, width, index, bounce, hashed, seed, logspp;
  int pattern;
  uint4 s0;
  MTD V2 structured(uint32_t dim) const {
    uint32_t pixelID = px + py * width;
    uint32_t sd = sampleSeed(sampleSeed(pixelID, dim), seed);
    uint32_t idx = index;
    if (pattern == 1) {
      uint32_t lg = logspp;
      if (idx == 0u) lg = 0u; else idx -= 1u;
      uint32_t block = idx >> lg;
      uint32_t mask = (1u << lg) - 1u;
      uint32_t morton = (morton2(px, py) << lg) | (idx & mask);
      idx = zSobolIndex(morton, dim, lg);
      sd = sampleSeed(sampleSeed(dim, seed), sampleSeed(px >> 8, py >> 8));
      if (index != 0u) block += 1u;
      sd = sampleSeed(sd, block);
    }
    uint32_t i = owen(idx, sampleSeed(sd, 0u));
    uint32_t x = __brev(lkPermute(i, sampleSeed(sd, 1u)));
    uint32_t y = owen(sobolD1(i), sampleSeed(sd, 2u));
    float fx = float(x >> 8) * (1.0f / 16777216.0f);
    float fy = float(y >> 8) * (1.0f / 16777216.0f);
    return {EPS + 0.999f * fx, EPS + 0.999f * fy};
  }
  MTD float rnd() {
    s0.x = s0.x * 1664525u + 1013904223u; s0.y = s0.y * 1664525u + 1013904223u;
    s0.z = s0.z * 1664525u + 1013904223u; s0.w = s0.w * 1664525u + 1013904223u;
    s0.x += s0.y * s0.w; s0.y += s0.z * s0.x; s0.z += s0.x * s0.y; s0.w += s0.y * s0.z;
    s0.x ^= s0.x >> 16; s0.y ^= s0.y >> 16; s0.z ^= s0.z >> 16; s0.w ^= s0.w >> 16;
    s0.x += s0.y * s0.w; s0.y += s0.z * s0.x; s0.z += s0.x * s0.y; s0.w += s0.y * s0.z;
    return float(s0.x) / float(0xffffffffu);
  }
  MTD float s1(uint32_t dim) {
    if (pattern == 2) return EPS + 0.999f * rnd();
    return structured(dim).x;
  }
  MTD V2 s2(uint32_t dim) {
    if (pattern == 2) { float a = s1(dim); float b = s1(dim); return {a, b}; }
    return structured(dim);
  }
  MTD float hashedSample(uint32_t slot) {
    uint32_t dim = sampleSeed(sampleSeed(bounce, slot), hashed) | 0x80000000u;
    hashed += 1u;
    if (pattern == 2) return EPS + 0.999f * rnd();
    uint32_t pixelID = px + py * width;
    uint32_t sd = sampleSeed(sampleSeed(pixelID, dim), seed);
    uint32_t i = owen(index, sampleSeed(sd, 0u));
    uint32_t x = __brev(lkPermute(i, sampleSeed(sd, 1u)));
    return EPS + 0.999f * (float(x >> 8) * (1.0f / 16777216.0f));
  }
  MTD float lightCandidateRandom(uint32_t salt) {
    if (pattern == 2) (void)rnd();
    uint32_t pixelID = px + py * width;
    uint32_t key = sampleSeed(sampleSeed(pixelID, index), seed);
    uint32_t dimension = sampleSeed(bounce, salt) ^ 0xa511e9b3u;
    return float(sampleHash(key ^ dimension) >> 8) * (1.0f / 16777216.0f);
  }
  MTD uint32_t bounceDim(uint32_t slot) const { return 3u + 8u + bounce * 64u + slot; }
  MTD uint32_t lightDim(uint32_t c, uint32_t slot) const {
    if (c == 0u) return slot == 2u ? bounceDim(8u) : bounceDim(slot);
    return bounceDim(9u + (c - 1u) * 3u + slot);
  }
};

// ---------------------------------------------------------------- traversal
// intersect.wgsl.ts:1500-1521 (every operation rounded, fminf/fmaxf)
MTD V3 traversalInverse(V3 d) { return {__frcp_rn(d.x), __frcp_rn(d.y), __frcp_rn(d.z)}; }
MTD float intersectBox(V3 o, V3 bmin, V3 bmax, V3 invD, float tMax) {
  V3 tBot = xmul3(xsub3(bmin, o), invD);
  V3 tTop = xmul3(xsub3(bmax, o), invD);
  float t0 = fmaxf(fminf(tBot.x, tTop.x), fmaxf(fminf(tBot.y, tTop.y), fminf(tBot.z, tTop.z)));
  float t1 = fminf(fmaxf(tBot.x, tTop.x), fminf(fmaxf(tBot.y, tTop.y), fmaxf(tBot.z, tTop.z)));
  if (t0 > t1 || t0 > tMax) return -1.0f;
  return t0 > 0.0f ? t0 : t1;
}
MTD int maxDimension(V3 v) {
  if (v.x > v.y) return v.x > v.z ? 0 : 2;
  return v.y > v.z ? 1 : 2;
}
// intersect.wgsl.ts:1430-1493; returns t (0 for a miss) and barycentrics.
MTD float intersectTriangle(V3 o, V3 p0, V3 p1, V3 p2, int maxDim, V3 shear, float tMax, V3 &bary) {
  V3 a = xsub3(p0, o), b = xsub3(p1, o), c = xsub3(p2, o);
  if (maxDim == 0) { a = {a.y, a.z, a.x}; b = {b.y, b.z, b.x}; c = {c.y, c.z, c.x}; }
  else if (maxDim == 1) { a = {a.z, a.x, a.y}; b = {b.z, b.x, b.y}; c = {c.z, c.x, c.y}; }
  a.x = xa(a.x, xm(shear.x, a.z)); a.y = xa(a.y, xm(shear.y, a.z));
  b.x = xa(b.x, xm(shear.x, b.z)); b.y = xa(b.y, xm(shear.y, b.z));
  c.x = xa(c.x, xm(shear.x, c.z)); c.y = xa(c.y, xm(shear.y, c.z));
  V3 e = {xs(xm(b.x, c.y), xm(b.y, c.x)), xs(xm(c.x, a.y), xm(c.y, a.x)), xs(xm(a.x, b.y), xm(a.y, b.x))};
  bool anyNeg = e.x < 0.0f || e.y < 0.0f || e.z < 0.0f;
  bool anyPos = e.x > 0.0f || e.y > 0.0f || e.z > 0.0f;
  if (anyNeg && anyPos) return 0.0f;
  float det = xa(xa(e.x, e.y), e.z);
  float az = xm(a.z, shear.z), bz = xm(b.z, shear.z), cz = xm(c.z, shear.z);
  float tScaled = xa(xa(xm(e.x, az), xm(e.y, bz)), xm(e.z, cz));
  if (fabsf(tScaled) > fabsf(xm(tMax, det))) return 0.0f;
  float invDet = __frcp_rn(det);
  bary = {xm(e.x, invDet), xm(e.y, invDet), xm(e.z, invDet)};
  return xm(tScaled, invDet);
}

MTD V3 vertexPosition(const DevScene &s, int32_t i) {
  const uint32_t *w = s.attr + size_t(i) * s.vstride;
  if (s.vstride == 4) {
    float4 q = __ldg(reinterpret_cast<const float4 *>(w));
    return {q.x, q.y, q.z};
  }
  return {asf(__ldg(w)), asf(__ldg(w + 1)), asf(__ldg(w + 2))};
}
// vertexAttributes.wgsl.ts:14-28
MTD V3 vertexNormal(const DevScene &s, int32_t i) {
  const uint32_t *w = s.attr + size_t(i) * s.vstride + s.vnormalOff;
  if (s.vnormalFloat) return {asf(__ldg(w)), asf(__ldg(w + 1)), asf(__ldg(w + 2))};
  uint32_t word = __ldg(w);
  int32_t a = int32_t(word << 16) >> 16;
  int32_t b = int32_t(word) >> 16;
  if (a == -32768 && b == -32768) return v3(0.0f);
  V3 v = {float(a) / 32767.0f, float(b) / 32767.0f, 0.0f};
  v.z = 1.0f - fabsf(v.x) - fabsf(v.y);
  if (v.z < 0.0f) {
    float nx = (1.0f - fabsf(v.y)) * (v.x >= 0.0f ? 1.0f : -1.0f);
    float ny = (1.0f - fabsf(v.x)) * (v.y >= 0.0f ? 1.0f : -1.0f);
    v.x = nx; v.y = ny;
  }
  return normalize(v);
}

// ------------------------------------------------------------ material maps
// materialBuffer.wgsl.ts:316-378 wrapMapCoordinate / sampleMap / loadMapTexel
// with independent textures.  The shader filters footprints inside the image
// in hardware and repeat footprints that cross its edge by hand; both are the
// bilinear mix of the four texels around wrapped * size - 0.5 with clamped
// (repeat: modular) texel coordinates, evaluated here in software for every
// footprint.  Rounded operations throughout (no contraction), so a lookup is
// bit-identical to the CPU restatement.
MTD float wrapMapCoordinate(float v, float mode) {
  if (mode < 0.5f) return __fsub_rn(v, floorf(v));
  if (mode < 1.5f) return clampf(v, 0.0f, 1.0f);
  const float m = __fsub_rn(v, __fmul_rn(2.0f, floorf(__fmul_rn(v, 0.5f))));
  return __fsub_rn(1.0f, fabsf(__fsub_rn(1.0f, m)));
}
static __device__ __noinline__ float4 sampleMap(const DevScene &s, int idx, V2 uv) {
  if (idx < 0 || uint32_t(idx) >= s.mapCount) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  const float4 *mi = s.maps + size_t(idx) * MTC_MAP_VEC4_ROWS;
  const float4 a = ld4(mi), t = ld4(mi + 1), modes = ld4(mi + 2);
  const int w = asi(a.x), h = asi(a.y);
  const uint32_t first = asu(a.z);
  if (w < 1 || h < 1 || uint64_t(first) + uint64_t(w) * uint64_t(h) > s.mapTexelCount)
    return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  const float tx = __fsub_rn(__fmul_rn(wrapMapCoordinate(__fadd_rn(__fmul_rn(uv.x, t.x), t.z), modes.z), float(w)), 0.5f);
  const float ty = __fsub_rn(__fmul_rn(wrapMapCoordinate(__fadd_rn(__fmul_rn(uv.y, t.y), t.w), modes.w), float(h)), 0.5f);
  const float fx = floorf(tx), fy = floorf(ty), wx = __fsub_rn(tx, fx), wy = __fsub_rn(ty, fy);
  // Finite coordinates wrap into [-1, size - 1]; the clamp only pins NaN.
  const int bx = int(fminf(fmaxf(fx, -1.0f), float(w))), by = int(fminf(fmaxf(fy, -1.0f), float(h)));
  auto load = [&](int x, int y) {
    int px = modes.z < 0.5f ? ((x % w) + w) % w : min(max(x, 0), w - 1);
    int py = modes.w < 0.5f ? ((y % h) + h) % h : min(max(y, 0), h - 1);
    return ld4(s.mapTexels + first + size_t(py) * size_t(w) + size_t(px));
  };
  const float4 t00 = load(bx, by), t10 = load(bx + 1, by), t01 = load(bx, by + 1), t11 = load(bx + 1, by + 1);
  auto mix1 = [](float p, float q, float k) { return __fadd_rn(__fmul_rn(p, __fsub_rn(1.0f, k)), __fmul_rn(q, k)); };
  auto mix4 = [&](float4 p, float4 q, float k) {
    return make_float4(mix1(p.x, q.x, k), mix1(p.y, q.y, k), mix1(p.z, q.z, k), mix1(p.w, q.w, k));
  };
  return mix4(mix4(t00, t10, wx), mix4(t01, t11, wx), wy);
}
// projectUV (uvProjection.wgsl.ts): procedural UVs from a local-space
// position and normal; 1 spherical, 2 cylindrical, 3 triplanar.
MTD V2 projectUV(int type, V3 pos, V3 normal) {
  if (type == 3) {
    const V3 a = {fabsf(normal.x), fabsf(normal.y), fabsf(normal.z)};
    if (a.x > a.y && a.x > a.z) return {pos.y, pos.z};
    if (a.y > a.x && a.y > a.z) return {pos.x, pos.z};
    return {pos.x, pos.y};
  }
  if (type == 1) {
    const V3 n = normalize(pos);
    return {atan2f(n.x, n.z) / (2.0f * PI) + 0.5f, 1.0f - acosf(n.y) / PI};
  }
  if (type == 2) return {atan2f(pos.z, pos.x) / (2.0f * PI) + 0.5f, pos.y};
  return {0.0f, 0.0f};
}

// A material's map index names a map of this scene (an index past the map
// table, like -1, means no map).
MTD bool mapValid(const DevScene &s, float index) { return index >= 0.0f && index < float(s.mapCount); }

// intersectionAlphaPasses (intersectionAlpha.wgsl.ts:14-90): whether a shadow
// ray's candidate hit on a triangle of `material` occludes.  Coverage is the
// material's alpha times the base color's alpha (map alpha usage "alpha") and
// the alpha map's g at the hit's UV, then resolved by the alpha mode: opaque
// occludes, mask compares with the cutoff, blend draws hashedSample(1).
static __device__ __noinline__ bool alphaPasses(const DevScene &s, int32_t material, int32_t record, int32_t i0,
                                                int32_t i1, int32_t i2, V3 bary, V3 hitPosition, V3 hitNormal,
                                                Sampler &smp) {
  if (s.triMats) {  // triangleMaterial (vertexAttributes.wgsl.ts:51-56)
    const uint32_t m = __ldg(s.triMats + record);
    if (m && m - 1u < s.matCount) material = int32_t(m - 1u);
  }
  const float4 *d = s.mats + size_t(material) * MTC_MATERIAL_VEC4_ROWS;
  const float4 r2 = ld4(d + 2), r5 = ld4(d + 5), r22 = ld4(d + 22);
  float alpha = ld4(d + 9).x;
  const bool baseAlpha = r5.w == 2.0f && mapValid(s, r2.z), alphaMap = mapValid(s, r22.z);
  if (baseAlpha || alphaMap) {
    V2 uv0 = {0.0f, 0.0f}, uv1 = uv0, uv2 = uv0;
    if (s.vuvOff) {
      auto vuv = [&](int32_t i) {
        const uint32_t *w = s.attr + size_t(i) * s.vstride + s.vuvOff;
        return V2{asf(__ldg(w)), asf(__ldg(w + 1))};
      };
      uv0 = vuv(i0); uv1 = vuv(i1); uv2 = vuv(i2);
    }
    const float4 r7 = ld4(d + 7);
    const int projection = int(r7.x);
    V2 uv = {bary.x * uv0.x + bary.y * uv1.x + bary.z * uv2.x, bary.x * uv0.y + bary.y * uv1.y + bary.z * uv2.y};
    if (projection > 0) uv = projectUV(projection, hitPosition, hitNormal);
    uv = {uv.x * r7.z, uv.y * r7.w};
    if (projection == 3) uv = {uv.x - floorf(uv.x), uv.y - floorf(uv.y)};
    if (baseAlpha) alpha *= sampleMap(s, int(r2.z), uv).w;
    if (alphaMap) alpha *= sampleMap(s, int(r22.z), uv).y;
  }
  const int mode = int(ld4(d + 23).w);
  if (mode == 0) alpha = 1.0f;
  else if (mode == 1) alpha = alpha >= r22.w ? 1.0f : 0.0f;
  if (mode == 2) return smp.hashedSample(1u) <= alpha;
  return alpha >= 1.0f;
}

struct TraversalHit {
  float tMax;
  V3 hitNormal, hitBary;
  int32_t triangleIndex, insIdx;
};

// getBVHTraverseCode (intersect.wgsl.ts:213-629) as a restartable state
// machine, for warps that keep a queue of rays and give a lane a new ray as
// soon as its current one has finished.  A lane's next piece of work is a
// node to visit (interior, either level), an instance of the open TLAS leaf
// to enter, or the triangles of a BLAS leaf; advance() runs one of these at a
// time for all lanes of the warp that are at it.  A lane that waits only
// waits: each ray's visit order, box tests, `>` tie rule and self-hit and
// backface rules are those of the reference's loop, so the hits are bit-identical
// to its.
//
// What bounds it is issue slots at few active lanes.  With every lane taking
// whatever step came next, an iteration ran the node code for ~20 lanes, the
// instance code for ~6 and the triangle code for ~2, and the last two cost as
// much as the first: 1,070 warp instructions a ray at 8.8 active lanes on the
// instanced scene (1.45M bounce rays, 2.56 ms).  Repeating node visits while
// enough lanes need one, the header word kept with each stack entry, paired
// f32 box tests, and the shear of the watertight test computed at leaves
// (2.3 a ray) instead of instances entered (11.4): 733 at 12.4 lanes, 1.98 ms.
// Paired box tests alone are 6 % of the 1080p instanced render.
//
// Dense and sparse queues want different waits.  A warp with many rays behind
// it goes back to the lanes at instances and leaves once fewer than
// kNodeLanes are at nodes (12: 124 ms, 1: 130 ms for 8 samples of the 1080p
// instanced scene); with few rays a warp's own latency is what counts, and it
// finishes the node visits first (1: 31.3 ms, 12: 33.2 ms for the glass scene
// at 1280x720, 6.4 against 6.9 for a 333x217 image).  Making lanes at leaves
// and instances wait for company lost in both (8 and 4 lanes: 37 and 9 ms).
constexpr uint32_t kNodeLanes = 12;
constexpr uint32_t kDenseRays = 128;  // rays per warp from which kNodeLanes holds (64: the same within noise)
constexpr int kTraversalStackEntries = 2 * MTC_MAX_STACK;

// What a finished closest-hit query stores; the geometric normal is
// recomputed from the triangle by whoever needs it (hitNormal).
struct alignas(16) StoredHit {
  float tMax, bary[3];
  int32_t triangleIndex, insIdx, _pad[2];
};

// The candidate normal of the triangle test (intersect.wgsl.ts:1482-1493) for
// the accepted triangle of a hit.
MTD V3 hitNormal(const DevScene &s, int32_t triangleIndex, int32_t insIdx) {
  const int32_t vertexOffset = asi(ld4(s.ins + size_t(insIdx) * MTC_INSTANCE_VEC4_STRIDE).y);
  const float4 r = ld4(s.bvh + triangleIndex);
  const V3 p0 = vertexPosition(s, asi(r.x) + vertexOffset), p1 = vertexPosition(s, asi(r.y) + vertexOffset),
           p2 = vertexPosition(s, asi(r.z) + vertexOffset);
  return xnormalize(xcross(xsub3(p1, p0), xsub3(p2, p0)));
}

// The shear of the watertight test (intersect.wgsl.ts:1500-1521), the axes
// selected before the divisions so that lanes of different dominant axes divide
// together.
MTD V3 selectShear(V3 d, int maxDim) {
  const float z = maxDim == 0 ? d.x : maxDim == 1 ? d.y : d.z;
  const float x = maxDim == 0 ? d.y : maxDim == 1 ? d.z : d.x;
  const float y = maxDim == 0 ? d.z : maxDim == 1 ? d.x : d.y;
  return {xd(-x, z), xd(-y, z), __frcp_rn(z)};
}

// A query as its source hands it to a warp.
struct RayQuery {
  V3 o, d;
  float limit;             // tMax at the start
  int32_t tri, ins;        // the triangle a bounce leaves from (tri -1: none)
  uint32_t payload, scene; // the source's own number of the query; its scene
  bool doubleSided;
};

// Shared memory of one warp: a batch of queries fetched together (word k of
// entry e at pending[k][e]) and the world-space ray of each lane's query, off
// the registers that the node visits need.
struct WarpRays {
  float pending[14][32];
  float ray[9][32];
};

// Three-operand minimum and maximum, and packed pairs of f32 operations, of
// sm_100: each half rounds like the scalar instruction.
MTD float min3(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
MTD float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
MTD uint64_t pack2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
MTD void unpack2(uint64_t v, float &lo, float &hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
MTD uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
MTD uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// A ray prepared for box tests: -origin and 1 / direction.
struct BoxRay {
  uint64_t oxy, ixy;
  float oz, iz;
  MTD void set(V3 o, V3 inv) {
    oxy = pack2(-o.x, -o.y);
    oz = -o.z;
    ixy = pack2(inv.x, inv.y);
    iz = inv.z;
  }
  MTD V3 origin() const {
    V3 o;
    unpack2(oxy, o.x, o.y);
    return {-o.x, -o.y, -oz};
  }
};

// intersectBox with its result split up: the entry and exit distances of the
// slabs.  A box is hit when t0 <= min(t1, tMax) and t1 > 0; intersectBox then
// returns t0 if positive, else t1.  (A min or max of all three axes is NaN
// only when every axis is, for t0 and t1 alike: a miss in both forms.)
MTD void boxSlabs(const BoxRay &r, ulonglong2 lo, ulonglong2 hi, float &t0, float &t1) {
  float bx, by, bz, cx, cy, cz, ignored;
  unpack2(mul2(add2(lo.x, r.oxy), r.ixy), bx, by);
  unpack2(mul2(add2(hi.x, r.oxy), r.ixy), cx, cy);
  unpack2(lo.y, bz, ignored);
  unpack2(hi.y, cz, ignored);
  bz = xm(xa(bz, r.oz), r.iz);
  cz = xm(xa(cz, r.oz), r.iz);
  t0 = max3(fminf(bx, cx), fminf(by, cy), fminf(bz, cz));
  t1 = min3(fmaxf(bx, cx), fmaxf(by, cy), fmaxf(bz, cz));
}
MTD ulonglong2 ldNode(const float4 *p) { return __ldg(reinterpret_cast<const ulonglong2 *>(p)); }
MTD int32_t nodeWord(ulonglong2 v) { return int32_t(uint32_t(v.y >> 32)); }

template <bool shadow, bool kGpuLayout, bool kAlpha = false>
struct RayTraversal {
  const DevScene *scene;
  const float4 *bvh;
  int32_t blasBase;
  float *world;  // rayO, rayD, 1 / rayD: word k at world[32 * k]
  // The ray of the level being visited (world, or the open instance's), the
  // instance-space direction, and what child pointers are relative to.
  BoxRay ray;
  V3 d;
  int32_t rel;
  int32_t currentTri, currentIns;
  bool doubleSided;
  // Node entries (index, header word) of the TLAS, those of the open instance
  // above them from `floor` on.  The array belongs to the caller (a local
  // array of the kernel): a dynamically indexed array inside this object
  // would keep the whole object, ray and hit included, in local memory.  Each
  // level is bounded by the reference's stack depth.
  int2 *stack;
  int top, floor;
  // What is worked on next: the node `cur` with its header word `ptr`.  An
  // interior node has ptr >= 0; else the state tells a TLAS leaf (-ptr
  // entries, or kEntriesLeft plus those an instance left to enter) from a
  // BLAS leaf.
  static constexpr int32_t kEntriesLeft = -(1 << 30);
  int32_t cur, ptr;
  enum : uint32_t { kTlas, kBlas, kDone, kIdle } state;
  int32_t leafNode, io;   // open TLAS leaf and its last entry still to enter
  int32_t vertexOffset, insIdx;
  bool gpuNodes;          // the open instance's BLAS is BVH_GPU
  float tMax;
  V3 bary;
  int32_t hitTri, hitIns;
  // Shadow queries of scenes with alpha: the path's sampler for alphaPasses,
  // and the query's tMax to restore after a hit that does not occlude.
  Sampler *alphaSmp;
  float tMaxInit;

  MTD bool found() const { return hitTri >= 0; }
  MTD V3 word3(int k) const { return {world[32 * k], world[32 * (k + 1)], world[32 * (k + 2)]}; }
  MTD bool atNode() const { return ptr >= 0; }
  MTD bool atLeaf() const { return ptr < 0 && state == kBlas; }
  MTD bool atInstances() const { return ptr < 0 && state == kTlas; }
  MTD void finish(uint32_t s) {
    state = decltype(state)(s);
    ptr = -1;
  }

  // Starts a query whose ray (`i` its inverse direction) passed the root box;
  // `column` is the lane's column of its warp's world-space rays.
  MTD void begin(const DevScene &s, int32_t base, float *column, V3 ro, V3 rd, V3 i, float limit, int32_t tri,
                 int32_t ins, bool bothSides) {
    scene = &s; bvh = s.bvh; blasBase = base;
    world = column;
    const float w[9] = {ro.x, ro.y, ro.z, rd.x, rd.y, rd.z, i.x, i.y, i.z};
#pragma unroll
    for (int k = 0; k < 9; k++) world[32 * k] = w[k];
    ray.set(ro, i);
    tMax = limit;
    currentTri = tri;
    currentIns = ins;
    doubleSided = bothSides;
    if (kAlpha) {
      alphaSmp = nullptr;
      tMaxInit = limit;
    }
    bary = v3(0.0f);
    hitTri = -1; hitIns = -1;
    gpuNodes = false;
    rel = 0; top = 0; floor = 0;
    state = kTlas;
    cur = 0;
    ptr = asi(ld4(bvh).w);
  }

  // Takes the next node off the stack; at the end of an instance, what is
  // left of its TLAS leaf (enter() goes on from there).
  MTD void pop() {
    if (top > floor) {
      const int2 e = stack[--top];
      cur = e.x;
      ptr = e.y;
    } else if (state == kBlas) {
      state = kTlas;
      cur = leafNode;
      ptr = kEntriesLeft + io + 1;
    } else {
      finish(kDone);
    }
  }

  // The interior visit at either level (intersect.wgsl.ts:265-300, :439-624):
  // box-test both children and go on with the one the reference pushes last
  // (the nearer, by the `>` rule), the other one on the stack.
  MTD void visit() {
    int32_t left = cur + 2, right = ptr + rel;
    ulonglong2 lmin, lmax, rmin, rmax;
    int32_t lptr, rptr;
    if (kGpuLayout && gpuNodes) {
      // BVH_GPU (BLAS layout 2, intersect.wgsl.ts:453-497): both child boxes
      // in the node, which may itself be a leaf.
      lmin = ldNode(bvh + cur);
      lmax = ldNode(bvh + cur + 1);
      rmin = ldNode(bvh + cur + 2);
      rmax = ldNode(bvh + cur + 3);
      const int32_t count = nodeWord(rmin);
      if (count > 0) {
        cur = rel + nodeWord(rmax) - 2;  // records at cur + 2
        ptr = -count;
        return;
      }
      left = rel + nodeWord(lmin) * 4;
      right = rel + nodeWord(lmax) * 4;
      lptr = rptr = 0;
    } else {
      lmin = ldNode(bvh + left);
      lmax = ldNode(bvh + left + 1);
      rmin = ldNode(bvh + right);
      rmax = ldNode(bvh + right + 1);
      lptr = nodeWord(lmin);
      rptr = nodeWord(rmin);
    }
    float l0, l1, r0, r1;
    boxSlabs(ray, lmin, lmax, l0, l1);
    boxSlabs(ray, rmin, rmax, r0, r1);
    const bool hitL = !(l0 > fminf(l1, tMax)) && l1 > 0.0f, hitR = !(r0 > fminf(r1, tMax)) && r1 > 0.0f;
    // The farther child is pushed first; without room for a second entry it
    // is the only one.
    const bool both = hitL && hitR, leftFar = (l0 > 0.0f ? l0 : l1) > (r0 > 0.0f ? r0 : r1);
    const bool push = both && top - floor + 1 < MTC_MAX_STACK;
    const bool nextLeft = both ? leftFar != push : hitL;
    if (push) stack[top++] = leftFar ? make_int2(left, lptr) : make_int2(right, rptr);
    cur = nextLeft ? left : right;
    ptr = nextLeft ? lptr : rptr;
    if (!(hitL || hitR)) pop();
  }

  // Next instance entry of the open TLAS leaf (descending, as the WGSL's
  // leaf loop): the ray in instance space, its BLAS root taken.  Without one,
  // the next TLAS node.
  MTD void enter() {
    if (ptr < kEntriesLeft / 2) {  // an instance was finished
      io = ptr - kEntriesLeft - 1;
    } else {
      leafNode = cur;
      io = -ptr - 1;
    }
    if (io < 0) {
      floor = 0;
      rel = 0;
      gpuNodes = false;
      ray.set(word3(0), word3(6));
      pop();
      return;
    }
    const float4 rec = ld4(bvh + leafNode + 2 + io);
    io--;
    insIdx = asi(rec.x);
    const float4 *insv = scene->ins + size_t(insIdx) * MTC_INSTANCE_VEC4_STRIDE;
    const float4 insData = ld4(insv);
    const float4 c0 = ld4(insv + 1), c1 = ld4(insv + 2), c2 = ld4(insv + 3), c3 = ld4(insv + 4);
    cur = asi(rec.y) + blasBase;
    const uint32_t encoded = asu(insData.x), layout = encoded >> 30;
    floor = top;
    if (layout != 0u && !(kGpuLayout && layout == 2u)) {  // TinyBVH bvh4 / cwbvh are not consumed
      cur = leafNode;
      ptr = kEntriesLeft + io + 1;
      return;
    }
    gpuNodes = kGpuLayout && layout == 2u;
    ptr = gpuNodes ? 0 : asi(ld4(bvh + cur).w);
    d = xmat4(c0, c1, c2, c3, word3(3), 0.0f);
    ray.set(xmat4(c0, c1, c2, c3, word3(0), 1.0f), traversalInverse(d));
    rel = blasBase + int32_t(encoded & 0x3fffffffu);
    vertexOffset = asi(insData.y);
    state = kBlas;
  }

  // The triangles of a BLAS leaf.
  MTD void leaf() {
    const int maxDim = maxDimension(vabs(d));
    const V3 shear = selectShear(d, maxDim), o = ray.origin();
    const int32_t last = cur + 2 - ptr;
    for (int32_t triangleIndex = cur + 2; triangleIndex < last; triangleIndex++) {
      if (triangleIndex == currentTri && insIdx == currentIns) continue;
      const float4 r = ld4(bvh + triangleIndex);
      const int32_t i0 = asi(r.x) + vertexOffset, i1 = asi(r.y) + vertexOffset, i2 = asi(r.z) + vertexOffset;
      const V3 p0 = vertexPosition(*scene, i0), p1 = vertexPosition(*scene, i1), p2 = vertexPosition(*scene, i2);
      V3 b;
      const float t = intersectTriangle(o, p0, p1, p2, maxDim, shear, tMax, b);
      if (!(t > 0.0f)) continue;
      if (!shadow && !doubleSided) {
        const int32_t material = asi(ld4(scene->ins + size_t(insIdx) * MTC_INSTANCE_VEC4_STRIDE).z) >> 8;
        const bool both = __ldg(&scene->mats[size_t(material) * MTC_MATERIAL_VEC4_ROWS + 23].z) > 0.5f;
        if (!both && xdot(xnormalize(xcross(xsub3(p1, p0), xsub3(p2, p0))), d) > 0.0f) continue;
      }
      tMax = t;
      if (shadow) {
        if (kAlpha && alphaSmp) {
          const int32_t material = asi(ld4(scene->ins + size_t(insIdx) * MTC_INSTANCE_VEC4_STRIDE).z) >> 8;
          if (!alphaPasses(*scene, material, triangleIndex, i0, i1, i2, b, o + d * t,
                           xnormalize(xcross(xsub3(p1, p0), xsub3(p2, p0))), *alphaSmp)) {
            tMax = tMaxInit;
            continue;
          }
        }
        hitTri = triangleIndex;
        finish(kDone);
        return;
      }
      bary = b;
      hitTri = triangleIndex;
      hitIns = insIdx;
    }
    pop();
  }

  // One round of the warp's busy lanes (all 32 lanes call it): leaves, then
  // instances, then at least one node visit and up to `steps` while
  // `nodeLanes` lanes need one.
  MTD void advance(uint32_t steps, uint32_t nodeLanes) {
    if (__any_sync(0xffffffffu, atLeaf())) {
      if (atLeaf()) leaf();
      __syncwarp();
    }
    if (__any_sync(0xffffffffu, atInstances())) {
      if (atInstances()) enter();
      __syncwarp();
    }
    unsigned node = __ballot_sync(0xffffffffu, atNode());
    for (uint32_t k = 0; node && k < steps; k++) {
      if (atNode()) visit();
      __syncwarp();
      node = __ballot_sync(0xffffffffu, atNode());
      if (uint32_t(__popc(node)) < nodeLanes) break;
    }
  }
};

// The root box test that starts every query.
MTD bool entersScene(const DevScene &s, V3 o, V3 inv, float limit) {
  return intersectBox(o, xyz(ld4(s.bvh)), xyz(ld4(s.bvh + 1)), inv, limit) > 0.0f;
}

// Drains a source's queries, numbered below `end`, with the calling warp (all
// 32 lanes call it).  The warp takes up to 32 queries at a time, every lane
// reading one of them, so that the chain of dependent loads behind a query
// (counter, queue, record, scene) is paid once a batch instead of by a whole
// warp at each lane's refill.
//
// The source has take(n): the number of the first of n queries that no one
// else gets; scene(i) and blasBase(i); read(t, query): false when query t is
// answered without a traversal; missed(query) for a ray past the root box,
// done(traversal, payload) for a finished one; and alpha(traversal, payload,
// scene) before a shadow query with coverage starts.
template <bool shadow, bool kGpuLayout, bool kAlpha, class Source>
MTD void traceQueue(Source &src, uint32_t end, uint32_t batch, uint32_t nodeLanes, uint32_t refillLanes,
                    uint32_t steps, WarpRays &rays) {
  int2 stack[kTraversalStackEntries];
  RayTraversal<shadow, kGpuLayout, kAlpha> rt;
  rt.stack = stack;
  rt.finish(rt.kIdle);
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t payload = 0, head = 0, have = 0;
  bool exhausted = false;
  for (;;) {
    const unsigned idle = __ballot_sync(0xffffffffu, rt.state == rt.kIdle);
    if (idle == 0xffffffffu && exhausted && head == have) break;
    // Refill once enough lanes wait (or none is left tracing).
    if (uint32_t(__popc(idle)) >= refillLanes || idle == 0xffffffffu) {
      if (head == have && !exhausted) {
        const uint32_t first = src.take(batch);
        exhausted = first >= end || end - first <= batch;
        RayQuery q;
        bool keep = lane < batch && first < end && lane < end - first && src.read(first + lane, q);
        V3 inv = v3(0.0f);
        if (keep) {
          inv = traversalInverse(q.d);
          if (!entersScene(src.scene(q.scene), q.o, inv, q.limit)) {
            src.missed(q);
            keep = false;
          }
        }
        const unsigned kept = __ballot_sync(0xffffffffu, keep);
        if (keep) {
          const uint32_t e = __popc(kept & ((1u << lane) - 1u));
          const float w[14] = {q.o.x, q.o.y, q.o.z, q.d.x, q.d.y, q.d.z, inv.x, inv.y, inv.z, q.limit,
                               __int_as_float(q.tri), __int_as_float(q.ins), __uint_as_float(q.payload),
                               __uint_as_float(q.scene | (q.doubleSided ? 0x80000000u : 0u))};
#pragma unroll
          for (int k = 0; k < 14; k++) rays.pending[k][e] = w[k];
        }
        __syncwarp();
        head = 0;
        have = __popc(kept);
      }
      const uint32_t e = head + __popc(idle & ((1u << lane) - 1u));
      if (rt.state == rt.kIdle && e < have) {
        float w[14];
#pragma unroll
        for (int k = 0; k < 14; k++) w[k] = rays.pending[k][e];
        payload = __float_as_uint(w[12]);
        const uint32_t i = __float_as_uint(w[13]) & 0x7fffffffu;
        rt.begin(src.scene(i), src.blasBase(i), &rays.ray[0][lane], {w[0], w[1], w[2]}, {w[3], w[4], w[5]},
                 {w[6], w[7], w[8]}, w[9], __float_as_int(w[10]), __float_as_int(w[11]),
                 __float_as_uint(w[13]) >> 31);
        if (kAlpha) src.alpha(rt, payload, i);
      }
      __syncwarp();
      head = min(have, head + uint32_t(__popc(idle)));
    }
    rt.advance(steps, nodeLanes);
    if (rt.state == rt.kDone) {
      src.done(rt, payload);
      rt.finish(rt.kIdle);
    }
    __syncwarp();
  }
}

}  // namespace mt
