// JGS2 step kernels for sm_100a.
//
// One frame of the stable Neo-Hookean Jacobi schedule runs as
//   prologue            predict + iteration-0 vertex frames + source preflight
//   per iteration:
//     solve             warp-cooperative per-vertex JGS2 local solve
//     gate              assembled determinant / energy reduction + accept
//     convergence       whole-pose revert, five-component residual, history,
//                       and the next iteration's vertex frames
//   epilogue            canonical copy, optional body correction, finalize
// which covers the reference's predict, tetPolarRotation, vertexPolarRotation,
// jgs2Solve, assembledVertexEnergy, candidateTetrahedron, reduceCandidate,
// applyCandidate, convergenceGradient, reduceConvergence, copyPosition,
// bodyHorizontalCorrection and finalize entry points
// (src/simulation/gpu/jgs2-shader.ts:2660-4589).  The graph-coloured schedule
// adds a copy and, per colour, a frame pass over the vertices that colour
// reads plus an in-place solve over the colour's vertices.
//
// Grid-wide reductions finish in the last block or warp to arrive (a ticket
// counter); sums are combined in a fixed order so results are deterministic.
// No kernel waits on another block.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "jgs2_cloth.cuh"
#include "jgs2_contact.cuh"
#include "jgs2_device.cuh"
#include "jgs2_kernels.cuh"

namespace jgs2 {
namespace {

constexpr int kBlock = 128;

// Checked build: device index checks in the gathers.  A failing check records
// its site once (the host reports it at the next synchronisation as
// JGS2_DEVICE_ERROR) and the gather skips the element, so the kernel never
// reads out of bounds.  Compiled out otherwise.
#ifndef JGS2_BOUNDS_CHECKS
#define JGS2_BOUNDS_CHECKS 0
#endif
enum BoundsSite : uint32_t {
  kSiteRecordTet = 1, kSiteRecordVertex = 2, kSiteIncidentTet = 3, kSiteTetVertex = 4, kSiteContactVertex = 5,
  kSiteListVertex = 6,
};
#if JGS2_BOUNDS_CHECKS
__device__ uint32_t gBoundsViolation;
#endif
__device__ __forceinline__ bool inBounds(uint64_t index, uint64_t limit, uint32_t site) {
#if JGS2_BOUNDS_CHECKS
  if (index < limit) return true;
  atomicCAS(&gBoundsViolation, 0u, site);
  return false;
#else
  (void)index; (void)limit; (void)site;
  return true;
#endif
}
__device__ __forceinline__ bool tetVerticesInBounds(const uint4& q, uint32_t V) {
  return inBounds(q.x, V, kSiteTetVertex) && inBounds(q.y, V, kSiteTetVertex) && inBounds(q.z, V, kSiteTetVertex) &&
         inBounds(q.w, V, kSiteTetVertex);
}
#ifndef JGS2_SOLVE_LANES
#define JGS2_SOLVE_LANES 4
#endif
// Lanes per vertex in the solve kernel.  A warp holds 32 / kGroup lane groups;
// a width that does not divide 32 leaves the warp's last lanes idle.
constexpr int kGroup = JGS2_SOLVE_LANES;
// Incident-tet gathers request the next tet's record before the current
// one's arithmetic (convergence, frames, the line search).
#ifndef JGS2_CONV_LOOKAHEAD
#define JGS2_CONV_LOOKAHEAD 1
#endif
constexpr int kRecFloats = 56;  // cached cubature record state

// Two float4 by one 256-bit load of data no kernel in flight writes, from a
// 32-byte boundary.  A gather's cost is its cache-line lookups, one per lane
// and instruction, not its bytes: a 64-byte record by two such loads takes
// half the lookups of four 128-bit ones.
__device__ __forceinline__ void load256(const float4* __restrict__ p, float4& a, float4& b) {
  asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
      : "l"(p));
}

struct TetRec {
  float3 g1, g2, g3;
  float vol, lambda, mu;
  uint4 idx;
};

__device__ __forceinline__ TetRec loadTet(const float4* __restrict__ tets, uint32_t t) {
  float4 a, b, c, d;
  load256(tets + 4ull * t, a, b);
  load256(tets + 4ull * t + 2, c, d);
  const uint4 q = make_uint4(__float_as_uint(d.x), __float_as_uint(d.y), __float_as_uint(d.z), __float_as_uint(d.w));
  TetRec r;
  r.g1 = f3(a.x, a.y, a.z);
  r.g2 = f3(b.x, b.y, b.z);
  r.g3 = f3(c.x, c.y, c.z);
  r.vol = a.w;
  r.lambda = b.w;
  r.mu = c.w;
  r.idx = q;
  return r;
}

// An incident-tet entry (tet * 4 + slot) and its record; false when a
// checked build finds the tet or one of its vertices out of range.
__device__ __forceinline__ bool incidentTetChecked(const float4* __restrict__ tets, uint32_t entry, uint32_t T,
                                                   uint32_t V, TetRec* r) {
  if (!inBounds(entry >> 2, T, kSiteIncidentTet)) return false;
  *r = loadTet(tets, entry >> 2);
  return tetVerticesInBounds(r->idx, V);
}

__device__ __forceinline__ float3 shapeGradient(const TetRec& r, uint32_t slot) {
  if (slot == 1) return r.g1;
  if (slot == 2) return r.g2;
  if (slot == 3) return r.g3;
  return -(r.g1 + r.g2 + r.g3);
}

__device__ __forceinline__ uint32_t idxAt(const uint4& q, uint32_t l) {
  return l == 0 ? q.x : (l == 1 ? q.y : (l == 2 ? q.z : q.w));
}

__device__ __forceinline__ M3 deformation(const TetRec& r, float3 x0, float3 x1, float3 x2, float3 x3) {
  return outer(x1 - x0, r.g1) + outer(x2 - x0, r.g2) + outer(x3 - x0, r.g3);
}

__device__ __forceinline__ M3 deformationAt(const TetRec& r, const float4* __restrict__ x) {
  return deformation(r, xyz(x[r.idx.x]), xyz(x[r.idx.y]), xyz(x[r.idx.z]), xyz(x[r.idx.w]));
}

__device__ __forceinline__ M3 loadRot(const float4* __restrict__ rot, uint32_t v) {
  const float4 a = rot[3ull * v], b = rot[3ull * v + 1], c = rot[3ull * v + 2];
  return {f3(a.x, a.y, a.z), f3(b.x, b.y, b.z), f3(c.x, c.y, c.z)};
}

// Reads of arrays that other blocks of the same launch may write (positions
// and vertex frames inside the persistent coloured sweep): kCoherent loads are
// ordinary weak loads (ld.global.ca), which the grid barrier's release and
// acquire fences order after the other blocks' writes; they never take the
// non-coherent read-only path (ld.global.nc), which a const __restrict__
// pointer may select and which no fence orders.  Other launches read these
// arrays as read-only data.
template <bool kCoherent>
__device__ __forceinline__ float4 ldPos(const float4* p, size_t i) {
  if constexpr (kCoherent) return __ldca(p + i);
  else return p[i];
}
template <bool kCoherent>
__device__ __forceinline__ M3 loadFrameT(const float4* pack, uint32_t v) {
  if constexpr (kCoherent) {
    const float4 a = __ldca(pack + 4ull * v), b = __ldca(pack + 4ull * v + 1), c = __ldca(pack + 4ull * v + 2);
    return {f3(a.x, a.y, a.z), f3(b.x, b.y, b.z), f3(c.x, c.y, c.z)};
  } else {
    const float4 a = pack[4ull * v], b = pack[4ull * v + 1], c = pack[4ull * v + 2];
    return {f3(a.x, a.y, a.z), f3(b.x, b.y, b.z), f3(c.x, c.y, c.z)};
  }
}
template <bool kCoherent>
__device__ __forceinline__ M3 deformationAtT(const TetRec& r, const float4* x) {
  if constexpr (kCoherent)
    return deformation(r, xyz(__ldca(x + r.idx.x)), xyz(__ldca(x + r.idx.y)), xyz(__ldca(x + r.idx.z)),
                       xyz(__ldca(x + r.idx.w)));
  else
    return deformationAt(r, x);
}

__device__ __forceinline__ void storeRot(float4* __restrict__ rot, uint32_t v, const M3& m) {
  rot[3ull * v] = make_float4(m.c0.x, m.c0.y, m.c0.z, 0.f);
  rot[3ull * v + 1] = make_float4(m.c1.x, m.c1.y, m.c1.z, 0.f);
  rot[3ull * v + 2] = make_float4(m.c2.x, m.c2.y, m.c2.z, 0.f);
}

// The frame of vertex v and its position at the same pose into the vertex's
// pack (its inertial target is the prologue's).
__device__ __forceinline__ void storeFrame(float4* __restrict__ pack, uint32_t v, const M3& m, float3 x) {
  pack[4ull * v] = make_float4(m.c0.x, m.c0.y, m.c0.z, x.x);
  pack[4ull * v + 1] = make_float4(m.c1.x, m.c1.y, m.c1.z, x.y);
  pack[4ull * v + 2] = make_float4(m.c2.x, m.c2.y, m.c2.z, x.z);
}
__device__ __forceinline__ M3 loadFrame(const float4* __restrict__ pack, uint32_t v) {
  return loadFrameT<false>(pack, v);
}

// What a record's tet needs of one of its vertices: frame, source position,
// inertial target and distributed inertia weight, 64 bytes in one place.
struct VertexPack {
  M3 R;
  float3 x, pred;
  float dW;
};
__device__ __forceinline__ VertexPack loadPack(const float4* __restrict__ pack, uint32_t v) {
  float4 a, b, c, d;
  load256(pack + 4ull * v, a, b);
  load256(pack + 4ull * v + 2, c, d);
  return {{xyz(a), xyz(b), xyz(c)}, f3(a.w, b.w, c.w), xyz(d), d.w};
}

// Row-major stored Ubar block l -> columns (cubatureBlock, jgs2-shader.ts:1204-1212).
// The record's 36 basis floats are 9 float4: floats [9l, 9l + 9) lie
// in the three float4 starting at (9l) / 4, so three vector loads replace nine
// scalar ones.  l must be a compile-time constant after unrolling.
__device__ __forceinline__ M3 loadBlockVec(const float4* __restrict__ rec, int l) {
  const int k0 = (9 * l) >> 2;
  const int off = 9 * l - 4 * k0;
  const float4 a = __ldg(rec + k0), b = __ldg(rec + k0 + 1), c = __ldg(rec + k0 + 2);
  const float f[12] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x, c.y, c.z, c.w};
  return {f3(f[off + 0], f[off + 3], f[off + 6]), f3(f[off + 1], f[off + 4], f[off + 7]),
          f3(f[off + 2], f[off + 5], f[off + 8])};
}

__device__ __forceinline__ uint32_t controlBits(float packed) {
  if (!finiteS(packed) || packed < 0.0f || packed > float(kControlMask) || packed != floorf(packed)) return 0u;
  return static_cast<uint32_t>(packed);
}

__device__ __forceinline__ bool latched(const DevParams& p, const FrameState* fs) {
  if (!p.stopEnabled) return false;
  return (controlBits(fs->control[0].w) & kStopLatchBit) != 0u;
}

__device__ __forceinline__ bool finiteNonnegInt(float v, float maximum) {
  return finiteS(v) && v >= 0.0f && v <= maximum && v == floorf(v);
}

__device__ __forceinline__ bool isPinned(const uint4& info) { return info.z != 0u; }

__device__ __forceinline__ ClothMaterial clothMaterial(const DevParams& p) {
  return {p.clothLambda, p.clothMu, p.clothThickness, p.clothBending};
}

__device__ __forceinline__ float distributedInertiaWeight(const float4& rm, const uint4& info, float invDt2) {
  if (isPinned(info)) return 0.0f;
  return rm.w * invDt2 / float(info.y > 1u ? info.y : 1u);
}

// vertexObjectiveGradient (jgs2-shader.ts:1926-1938).
__device__ __forceinline__ float3 objectiveGradient(const DevParams& p, const Buffers& b, uint32_t v, float3 pos) {
  float3 r = f3(0, 0, 0);
  if (p.objectiveFlags & 1u) r = r - xyz(b.forces[v]);
  if (p.objectiveFlags & 2u) {
    const float4 t = b.targets[v];
    if (t.w > 0.0f) r = r + t.w * (pos - xyz(t));
  }
  return r;
}

__device__ __forceinline__ float targetStiffness(const DevParams& p, const Buffers& b, uint32_t v) {
  return (p.objectiveFlags & 2u) ? b.targets[v].w : 0.0f;
}

// vertexObjectiveEnergyDelta (jgs2-shader.ts:1903-1924).
__device__ __forceinline__ float objectiveDelta(const DevParams& p, const Buffers& b, uint32_t v, float3 base,
                                                float3 d) {
  float r = 0.0f;
  if (p.objectiveFlags & 1u) r -= dot3(xyz(b.forces[v]), d);
  if (p.objectiveFlags & 2u) {
    const float4 t = b.targets[v];
    if (t.w > 0.0f) r += t.w * (dot3(base - xyz(t), d) + 0.5f * dot3(d, d));
  }
  return r;
}

__device__ __forceinline__ float floorDelta(const DevParams& p, float baseY, float dY) {
  if (!(p.floorStiffness > 0.0f)) return 0.0f;
  const float i = fminf(0.0f, baseY - p.floorHeight);
  const float f = fminf(0.0f, baseY + dY - p.floorHeight);
  return 0.5f * p.floorStiffness * (f - i) * (f + i);
}

// vertexImplicitEnergyAt without cloth/IPC terms (jgs2-shader.ts:2557-2645).
__device__ __forceinline__ float implicitEnergy(const DevParams& p, const Buffers& b, uint32_t v, float3 x,
                                                const uint4& info) {
  if (isPinned(info)) return 0.0f;
  const float4 rm = b.restMass[v];
  const float3 r = x - xyz(b.predicted[v]);
  float e = 0.5f * (rm.w * p.invDt2) * dot3(r, r);
  if (p.objectiveFlags != 0u) {
    if (p.objectiveFlags & 1u) e -= dot3(xyz(b.forces[v]), x);
    if (p.objectiveFlags & 2u) {
      const float4 t = b.targets[v];
      if (t.w > 0.0f) {
        const float3 q = x - xyz(t);
        e += 0.5f * t.w * dot3(q, q);
      }
    }
  }
  if (p.floorStiffness > 0.0f) {
    const float pen = fminf(0.0f, x.y - p.floorHeight);
    e += 0.5f * p.floorStiffness * pen * pen;
  }
  return e;
}

// Reductions over a lane group of W lanes inside one warp.  A power-of-two
// width folds with an xor butterfly; another width gathers the group's values
// in lane order on every lane, so all lanes hold the same, order-fixed result.
template <int W>
__device__ __forceinline__ uint32_t groupBase() {
  return ((threadIdx.x & 31u) / W) * W;
}
template <int W>
__device__ __forceinline__ float groupSum(float v, unsigned mask) {
  if constexpr ((W & (W - 1)) == 0) {
#pragma unroll
    for (int o = W / 2; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o, W);
    return v;
  } else {
    const uint32_t base = groupBase<W>();
    float s = __shfl_sync(mask, v, base);
#pragma unroll
    for (int j = 1; j < W; ++j) s += __shfl_sync(mask, v, base + j);
    return s;
  }
}
// Merge of the lanes' compensated sums over a lane group (xor butterfly;
// every lane ends with the same pair because the merge is symmetric).
template <int W>
__device__ __forceinline__ Comp3 shflComp(const Comp3& a, unsigned mask, uint32_t src) {
  Comp3 t;
  t.s.x = __shfl_sync(mask, a.s.x, src);
  t.s.y = __shfl_sync(mask, a.s.y, src);
  t.s.z = __shfl_sync(mask, a.s.z, src);
  t.c.x = __shfl_sync(mask, a.c.x, src);
  t.c.y = __shfl_sync(mask, a.c.y, src);
  t.c.z = __shfl_sync(mask, a.c.z, src);
  return t;
}
template <int W>
__device__ __forceinline__ void groupMerge(Comp3& a, unsigned mask) {
  if constexpr ((W & (W - 1)) == 0) {
#pragma unroll
    for (int o = W / 2; o > 0; o >>= 1) {
      Comp3 t;
      t.s.x = __shfl_xor_sync(mask, a.s.x, o, W);
      t.s.y = __shfl_xor_sync(mask, a.s.y, o, W);
      t.s.z = __shfl_xor_sync(mask, a.s.z, o, W);
      t.c.x = __shfl_xor_sync(mask, a.c.x, o, W);
      t.c.y = __shfl_xor_sync(mask, a.c.y, o, W);
      t.c.z = __shfl_xor_sync(mask, a.c.z, o, W);
      cmerge(a, t);
    }
  } else {
    const uint32_t base = groupBase<W>();
    Comp3 r = shflComp<W>(a, mask, base);
#pragma unroll
    for (int j = 1; j < W; ++j) cmerge(r, shflComp<W>(a, mask, base + j));
    a = r;
  }
}
template <int W>
__device__ __forceinline__ float groupMin(float v, unsigned mask) {
  if constexpr ((W & (W - 1)) == 0) {
#pragma unroll
    for (int o = W / 2; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(mask, v, o, W));
    return v;
  } else {
    const uint32_t base = groupBase<W>();
    float m = __shfl_sync(mask, v, base);
#pragma unroll
    for (int j = 1; j < W; ++j) m = fminf(m, __shfl_sync(mask, v, base + j));
    return m;
  }
}

// Deterministic block sum of doubles (fixed tree order).
template <int N>
__device__ __forceinline__ void blockSumDoubles(double (&vals)[N], double* scratch /* N * kBlock */) {
#pragma unroll
  for (int i = 0; i < N; ++i) scratch[i * kBlock + threadIdx.x] = vals[i];
  __syncthreads();
  for (int stride = kBlock / 2; stride > 0; stride >>= 1) {
    if (threadIdx.x < stride) {
#pragma unroll
      for (int i = 0; i < N; ++i)
        scratch[i * kBlock + threadIdx.x] += scratch[i * kBlock + threadIdx.x + stride];
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < N; ++i) vals[i] = scratch[i * kBlock];
}

// Exact incident block of the local Hessian for shape gradient g
// (jgs2-shader.ts:3097-3111): vol (a |g|^2 I + c1 u u^T + lambda w w^T) with
// u = F g and w = cof(F) g, the stable Neo-Hookean tangent applied to the
// rank-one direction e_i g^T.
__device__ __forceinline__ S3 incidentBlock(const TetRec& r, const M3& F, const PiolaTerms& pt, float3 g) {
  const float3 u1 = mv(F, g), w1 = mv(pt.cof, g);
  S3 blk = szero();
  saddDiag(blk, pt.a * dot3(g, g));
  saddOuter(blk, pt.c1, u1);
  saddOuter(blk, r.lambda, w1);
  return blk;
}
__device__ __forceinline__ void addIncidentBlock(S3& hess, const TetRec& r, const M3& F, const PiolaTerms& pt,
                                                 float3 g) {
  saddScaled(hess, r.vol, incidentBlock(r, F, pt, g));
}

__device__ __forceinline__ void storeIncident(float4* __restrict__ inc, uint32_t v, float3 g, const S3& h) {
  inc[3ull * v] = make_float4(g.x, g.y, g.z, h.xx);
  inc[3ull * v + 1] = make_float4(h.yy, h.zz, h.xy, h.xz);
  inc[3ull * v + 2] = make_float4(h.yz, 0.0f, 0.0f, 0.0f);
}

// Sums over a vertex's incident tets at one pose: the compensated material
// gradient sum vol P(F) g, the Hessian blocks, the volume-weighted F and the
// volume.
struct IncidentSums {
  Comp3 grad;
  S3 hess;
  M3 avg;
  float total;
};
__device__ __forceinline__ IncidentSums incidentZero() { return {czero(), szero(), mzero(), 0.0f}; }

// One thread per vertex: the tets in adjacency order, the next tet's record
// requested before the current one's arithmetic so its latency overlaps the
// work.
template <bool kHessian>
__device__ __forceinline__ void incidentSums(const Buffers& b, const float4* __restrict__ x, const uint4& info,
                                             IncidentSums& o) {
#if JGS2_CONV_LOOKAHEAD
  uint32_t nextEntry = info.y ? __ldg(&b.adjacency[info.x]) : 0u;
  TetRec nextRec;
  bool nextOk = false;
  if (info.y) nextOk = incidentTetChecked(b.tets, nextEntry, b.tetTotal, b.vertexTotal, &nextRec);
#endif
  for (uint32_t a = 0; a < info.y; ++a) {
#if JGS2_CONV_LOOKAHEAD
    const uint32_t entry = nextEntry;
    const TetRec r = nextRec;
    const bool tetOk = nextOk;
    if (a + 1 < info.y) {
      nextEntry = __ldg(&b.adjacency[info.x + a + 1]);
      nextOk = incidentTetChecked(b.tets, nextEntry, b.tetTotal, b.vertexTotal, &nextRec);
    }
#else
    const uint32_t entry = __ldg(&b.adjacency[info.x + a]);
    TetRec r;
    const bool tetOk = incidentTetChecked(b.tets, entry, b.tetTotal, b.vertexTotal, &r);
#endif
    if (!tetOk) continue;
    const M3 F = deformationAt(r, x);
    const PiolaTerms pt = piolaTerms(F, r.lambda, r.mu);
    const float3 g = shapeGradient(r, entry & 3u);
    cadd(o.grad, r.vol * mv(piola(F, pt), g));
    if (kHessian) addIncidentBlock(o.hess, r, F, pt, g);
    o.avg = o.avg + r.vol * F;
    o.total += r.vol;
  }
}

// Eight lanes per vertex, for scenes too small to hide a thread's chain of 24
// dependent tet gathers behind other warps: each lane evaluates one tet of a
// round into its row of `rows`, then the lanes add the rows in adjacency
// order, a few of the 19 sums each.  Every sum takes the same operands in the
// same order and with the same fused multiply-adds as incidentSums, so both
// give the same bits.  The sums go to `out` (kIncidentSum floats), from which
// one thread per vertex carries on, so that the polar iterations fill a warp
// instead of one lane of every group.
constexpr int kIncidentLanes = 8;
constexpr int kIncidentRow = 20;  // gradient 3, Hessian 6, F 9, 1, volume
constexpr int kIncidentGroup = kIncidentLanes * kIncidentRow + 8;  // floats per group; groups of a warp on different banks
constexpr int kIncidentSum = 23;  // 19 sums, 3 gradient compensations; odd, so vertices lie on different banks
constexpr int kWideBlock = kConvChunk * kIncidentLanes;  // a reduction entry's vertices
static_assert(kConvChunk == 32, "an entry's vertices are one warp");
struct IncidentShared {
  float4 rows4[kConvChunk * kIncidentGroup / 4];
  float sums[kConvChunk][kIncidentSum];
};
// What the sums are for: the frame alone, or the whole incident system too.
enum IncidentPart { kFramePart, kSystemPart };
template <IncidentPart kPart>
__device__ __forceinline__ void incidentSumsLanes(const Buffers& b, const float4* __restrict__ x, const uint4& info,
                                                  float* rows, uint32_t lane, unsigned mask, float* out,
                                                 uint4 cloth = make_uint4(0u, 0u, 0u, 0u),
                                                 const ClothMaterial& material = ClothMaterial{}) {
  float s[3] = {0.0f, 0.0f, 0.0f}, c = 0.0f;
  for (uint32_t a0 = 0; a0 < info.y; a0 += kIncidentLanes) {
    const uint32_t n = min(info.y - a0, static_cast<uint32_t>(kIncidentLanes));
    if (lane < n) {
      const uint32_t entry = __ldg(&b.adjacency[info.x + a0 + lane]);
      TetRec r;
      float row[kIncidentRow];
#pragma unroll
      for (int i = 0; i < kIncidentRow; ++i) row[i] = 0.0f;
      if (incidentTetChecked(b.tets, entry, b.tetTotal, b.vertexTotal, &r)) {
        const M3 F = deformationAt(r, x);
        if constexpr (kPart == kSystemPart) {
          const PiolaTerms pt = piolaTerms(F, r.lambda, r.mu);
          const float3 g = shapeGradient(r, entry & 3u);
          const float3 f = r.vol * mv(piola(F, pt), g);
          row[0] = f.x; row[1] = f.y; row[2] = f.z;
          const S3 blk = incidentBlock(r, F, pt, g);
          row[3] = blk.xx; row[4] = blk.yy; row[5] = blk.zz; row[6] = blk.xy; row[7] = blk.xz; row[8] = blk.yz;
        }
        row[9] = F.c0.x; row[10] = F.c0.y; row[11] = F.c0.z;
        row[12] = F.c1.x; row[13] = F.c1.y; row[14] = F.c1.z;
        row[15] = F.c2.x; row[16] = F.c2.y; row[17] = F.c2.z;
        row[18] = 1.0f;
        row[19] = r.vol;
      }
      float4* dst = reinterpret_cast<float4*>(rows + lane * kIncidentRow);
#pragma unroll
      for (int i = 0; i < kIncidentRow / 4; ++i)
        dst[i] = make_float4(row[4 * i], row[4 * i + 1], row[4 * i + 2], row[4 * i + 3]);
    }
    __syncwarp(mask);
    for (uint32_t j = 0; j < n; ++j) {
      const float* q = rows + j * kIncidentRow;
      const float vol = q[19];
      if (kPart == kSystemPart) {
        if (lane < 3) {
          float e;
          s[0] = twoSum(s[0], q[lane], &e);
          c = __fadd_rn(c, e);
        } else {
          s[0] = __fmaf_rn(vol, q[lane], s[0]);
        }
      }
      s[1] = __fmaf_rn(vol, q[8 + lane], s[1]);
      if (lane < 3) s[2] = __fmaf_rn(vol, q[16 + lane], s[2]);
    }
    __syncwarp(mask);
  }
  if constexpr (kPart == kSystemPart) {
    // The vertex's cloth triangles, then its hinges, a lane each likewise.
    for (uint32_t a0 = 0; a0 < cloth.y + cloth.w;) {
      const bool triangles = a0 < cloth.y;
      const uint32_t end = triangles ? cloth.y : cloth.y + cloth.w;
      const uint32_t n = min(end - a0, static_cast<uint32_t>(kIncidentLanes));
      if (lane < n) {
        float row[kClothRow];
        if (triangles)
          clothTriangleRow(b.clothTris, __ldg(&b.clothIncidence[cloth.x + a0 + lane]), x, material, row);
        else
          clothHingeRow(b.clothHinges, __ldg(&b.clothIncidence[cloth.z + a0 - cloth.y + lane]), x, material, row);
#pragma unroll
        for (int i = 0; i < kClothRow; ++i) rows[lane * kIncidentRow + i] = row[i];
      }
      __syncwarp(mask);
      for (uint32_t j = 0; j < n; ++j) {
        const float* q = rows + j * kIncidentRow;
        if (lane < 3) {
          float e;
          s[0] = twoSum(s[0], q[lane], &e);
          c = __fadd_rn(c, e);
        } else {
          s[0] = __fmaf_rn(q[lane], q[6 + lane], s[0]);
        }
        if (lane == 0) s[1] = __fmaf_rn(q[8], q[14], s[1]);
      }
      __syncwarp(mask);
      a0 += n;
    }
  }
  out[lane] = s[0];
  out[8 + lane] = s[1];
  if (lane < 3) {
    out[16 + lane] = s[2];
    out[19 + lane] = c;
  }
}
__device__ __forceinline__ IncidentSums loadIncidentSums(const float* q) {
  IncidentSums o;
  o.grad.s = f3(q[0], q[1], q[2]);
  o.grad.c = f3(q[19], q[20], q[21]);
  o.hess = {q[3], q[4], q[5], q[6], q[7], q[8]};
  o.avg = {f3(q[9], q[10], q[11]), f3(q[12], q[13], q[14]), f3(q[15], q[16], q[17])};
  o.total = q[18];
  return o;
}
// The sums of an entry's (at most 32) vertices, eight lanes per vertex, left
// in shared memory (ends with a block barrier).
__device__ __forceinline__ void incidentBlockSums(const Buffers& b, const DevParams& p, const float4* __restrict__ x,
                                                  const RedBlock& rb, const SceneRange& sr, bool pinnedToo,
                                                  IncidentShared& sh) {
  const uint32_t group = threadIdx.x / kIncidentLanes, k = rb.begin + group;
  if (k < rb.end) {
    const uint4 info = b.vinfo[sr.vOff + k];
    if (pinnedToo || !isPinned(info))
      incidentSumsLanes<kSystemPart>(b, x, info, reinterpret_cast<float*>(sh.rows4) + group * kIncidentGroup,
                                     threadIdx.x % kIncidentLanes, 0xffu << (threadIdx.x & 24u), sh.sums[group],
                                     p.cloth && !isPinned(info) ? b.clothRange[sr.vOff + k] : make_uint4(0u, 0u, 0u, 0u),
                                     clothMaterial(p));
  }
  __syncthreads();
}

// Cloth terms, frame and incident system of a free vertex from its sums: the
// frame is the polar of the volume-weighted average F (vertexPolarRotation,
// jgs2-shader.ts:2959-2989), the system the incident material gradient and
// Hessian blocks plus the membrane and bending terms of the vertex's cloth.
__device__ __forceinline__ void storeFrameAndIncident(const Buffers& b, const DevParams& p,
                                                      const float4* __restrict__ x, uint32_t v, const uint4& info,
                                                      IncidentSums& o, bool clothToo) {
  if (p.cloth && clothToo)
    clothLocalSystem<true>(b.clothTris, b.clothHinges, b.clothIncidence, b.clothRange[v], x, clothMaterial(p), 0u, 1u,
                           o.grad, o.hess);
  const M3 favg = o.total > 0.0f ? (1.0f / o.total) * o.avg : midentity();
  storeFrame(b.vertexPack, v, info.y == 0u ? midentity() : polarRotation(favg, p.rotationEpsilon), xyz(x[v]));
  storeIncident(b.incident, v, cvalue(o.grad), o.hess);
}

// Vertex frame: polar of the volume-weighted average F over incident tets
// (vertexPolarRotation, jgs2-shader.ts:2959-2989).
template <bool kCoherent = false>
__device__ __forceinline__ M3 vertexFrame(const Buffers& b, const float4* __restrict__ x, uint32_t v, float eps) {
  const uint4 info = b.vinfo[v];
  if (info.y == 0u) return midentity();
  M3 avg = mzero();
  float total = 0.0f;
  for (uint32_t a = 0; a < info.y; ++a) {
    const uint32_t entry = __ldg(&b.adjacency[info.x + a]);
    TetRec r;
    if (!incidentTetChecked(b.tets, entry, b.tetTotal, b.vertexTotal, &r)) continue;
    avg = avg + r.vol * deformationAtT<kCoherent>(r, x);
    total += r.vol;
  }
  avg = total > 0.0f ? (1.0f / total) * avg : midentity();
  return polarRotation(avg, eps);
}

// Vertex frames for a list of vertices (or all) from pose x.  kWide: eight
// lanes per vertex, 32 vertices a block, with the same bits, for lists of up
// to kWideVertices (a colour of a 525-vertex bar: 18.6 us one thread per
// vertex, 10.8 us so).
template <bool kWide>
__global__ void __launch_bounds__(kWide ? kWideBlock : kBlock) vertexPolarKernel(Buffers b,
                                                                                 const DevParams* __restrict__ pp,
                                                                                 const float4* __restrict__ x,
                                                                                 const uint32_t* __restrict__ list,
                                                                                 uint32_t count) {
  if constexpr (kWide) {
    __shared__ IncidentShared sh;
    const uint32_t group = threadIdx.x / kIncidentLanes, first = blockIdx.x * kConvChunk;
    auto wanted = [&](uint32_t i, uint32_t* v) {
      if (i >= count) return false;
      *v = list ? list[i] : i;
      const uint32_t scene = b.vertexScene[*v];
      return pp[scene].active && !latched(pp[scene], &b.frames[scene]);
    };
    uint32_t v;
    if (wanted(first + group, &v))
      incidentSumsLanes<kFramePart>(b, x, b.vinfo[v], reinterpret_cast<float*>(sh.rows4) + group * kIncidentGroup,
                                    threadIdx.x % kIncidentLanes, 0xffu << (threadIdx.x & 24u), sh.sums[group]);
    __syncthreads();
    if (threadIdx.x < kConvChunk && wanted(first + threadIdx.x, &v)) {
      const IncidentSums sums = loadIncidentSums(sh.sums[threadIdx.x]);
      const M3 avg = sums.total > 0.0f ? (1.0f / sums.total) * sums.avg : midentity();
      storeFrame(b.vertexPack, v,
                 b.vinfo[v].y == 0u ? midentity() : polarRotation(avg, pp[b.vertexScene[v]].rotationEpsilon),
                 xyz(x[v]));
    }
  } else {
    const uint32_t i = blockIdx.x * kBlock + threadIdx.x;
    if (i >= count) return;
    const uint32_t v = list ? list[i] : i;
    const uint32_t scene = b.vertexScene[v];
    const DevParams& p = pp[scene];
    if (!p.active || latched(p, &b.frames[scene])) return;
    storeFrame(b.vertexPack, v, vertexFrame(b, x, v, p.rotationEpsilon), xyz(x[v]));
  }
}

// ---------------------------------------------------------------------------
// Co-rotated linear path (the reference's legacy co-rotated branches of
// jgs2Solve and tetPolarRotation, jgs2-shader.ts:2931-2957, 2991-3263,
// 2479-2512).  No globalization: each vertex takes a regularised Newton step
// clamped to maxStep, and no gate or convergence pass follows.

// Tet frames: polar of each co-rotated tet's deformation gradient.
__global__ void __launch_bounds__(kBlock) tetPolarKernel(Buffers b, const DevParams* __restrict__ pp,
                                                         const float4* __restrict__ x, uint32_t T) {
  const uint32_t t = blockIdx.x * kBlock + threadIdx.x;
  if (t >= T) return;
  const DevParams& p = pp[b.tetScene[t]];
  if (!p.active) return;
  const TetRec r = loadTet(b.tets, t);
  storeRot(b.tetRot, t, polarRotation(deformationAt(r, x), p.rotationEpsilon));
}

// Block (rv, cv) of a tet's 12 x 12 row-major rest stiffness, as columns.
__device__ __forceinline__ M3 stiffnessBlock(const float* __restrict__ k, uint32_t rv, uint32_t cv) {
  const float* r0 = k + (3 * rv) * 12 + 3 * cv;
  const float* r1 = r0 + 12;
  const float* r2 = r1 + 12;
  return {f3(r0[0], r1[0], r2[0]), f3(r0[1], r1[1], r2[1]), f3(r0[2], r1[2], r2[2])};
}

// Displacements of a co-rotated tet's vertices in its frame,
// R^T (x_l - centroid) - (X_l - rest centroid).
__device__ __forceinline__ void corotatedDisplacement(const Buffers& b, const float4* __restrict__ x, const uint4& q,
                                                      const M3& R, float3 disp[4]) {
  float3 cur[4], rest[4];
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    const uint32_t v = idxAt(q, l);
    cur[l] = xyz(x[v]);
    rest[l] = xyz(b.restMass[v]);
  }
  const float3 cc = 0.25f * (cur[0] + cur[1] + cur[2] + cur[3]);
  const float3 rc = 0.25f * (rest[0] + rest[1] + rest[2] + rest[3]);
  const M3 Rt = mtrans(R);
#pragma unroll
  for (int l = 0; l < 4; ++l) disp[l] = mv(Rt, cur[l] - cc) - (rest[l] - rc);
}

// Block row `row` of a tet's rest stiffness: its four 3 x 3 blocks, from nine
// vector loads.
struct StiffnessRow {
  M3 block[4];
};
__device__ __forceinline__ StiffnessRow stiffnessRow(const float* __restrict__ k, uint32_t row) {
  const float4* q = reinterpret_cast<const float4*>(k) + 9u * row;
  float f[3][12];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const float4 v = __ldg(q + 3 * i + j);
      f[i][4 * j] = v.x; f[i][4 * j + 1] = v.y; f[i][4 * j + 2] = v.z; f[i][4 * j + 3] = v.w;
    }
  StiffnessRow r;
#pragma unroll
  for (int c = 0; c < 4; ++c)
    r.block[c] = {f3(f[0][3 * c], f[1][3 * c], f[2][3 * c]), f3(f[0][3 * c + 1], f[1][3 * c + 1], f[2][3 * c + 1]),
                  f3(f[0][3 * c + 2], f[1][3 * c + 2], f[2][3 * c + 2])};
  return r;
}

// R sum_c K_row,c d_c: a row of the element gradient (tetGradient) or of the
// rotated stiffness times one basis column.
__device__ __forceinline__ float3 stiffnessTimes(const StiffnessRow& row, const M3& R, const float3 d[4]) {
  float3 lg = f3(0, 0, 0);
#pragma unroll
  for (int c = 0; c < 4; ++c) lg = lg + mv(row.block[c], d[c]);
  return mv(R, lg);
}

// Element gradient of a co-rotated record's tet and its reduced Hessian
// (cubatureHessian), column c = sum_l B_l^T R K_l. R^T B_.[:, c], a block row of
// the stiffness at a time so that each of its 144 floats is loaded once.
__device__ __forceinline__ M3 corotatedRecordSystem(const float* __restrict__ k, const M3& R, const float3 disp[4],
                                                    const M3 basis[4], float3 tg[4]) {
  const M3 Rt = mtrans(R);
  float3 ld[3][4];
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    ld[0][l] = mv(Rt, basis[l].c0);
    ld[1][l] = mv(Rt, basis[l].c1);
    ld[2][l] = mv(Rt, basis[l].c2);
  }
  float3 col[3];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const StiffnessRow row = stiffnessRow(k, r);
    tg[r] = stiffnessTimes(row, R, disp);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float3 wp = stiffnessTimes(row, R, ld[c]);
      const float3 d = mtv(basis[r], wp);
      col[c] = r == 0 ? d : col[c] + d;
    }
  }
  return {col[0], col[1], col[2]};
}

// Distributed objective gradient / target stiffness of a record vertex.
__device__ __forceinline__ float3 distributedObjective(const DevParams& p, const Buffers& b, uint32_t q, float3 x,
                                                     const uint4& qi) {
  if (isPinned(qi)) return f3(0, 0, 0);
  return objectiveGradient(p, b, q, x) * (1.0f / float(qi.y > 1u ? qi.y : 1u));
}

// The exact co-rotated gather, the cubature complement and the regularised
// solve (regularizedSolve, :2479-2512) of kCoVertices vertices per block.
// Every incident tet and every record is one thread's item: its gradient (3)
// and Hessian (9) contribution goes to shared memory, then 12 threads per
// vertex add one component each over the items in order (the vertex's own
// terms, incident tets in adjacency order, floor, records in record order),
// and one thread per vertex solves.  Bound by the latency of an item's gathers
// and its 144-float stiffness, of which every float is loaded once, nine
// vector loads a block row.  One thread per vertex for all of it, as before,
// walked 24 tets and K records one after another and loaded the stiffness
// four times: 322 us per launch at 1 200 vertices (now 17), 340 at 9 020 (now
// 49).  The contributions and the order of the sums are the same, so are the
// bits.  Two blocks per SM (246 registers, no spills); three spill 220 bytes,
// gain 6 % at 9 020 vertices and lose 3 % at 1 200.
constexpr uint32_t kCoVertices = 10;   // 120 component sums on 128 threads
constexpr uint32_t kCoTets = 24;       // incident tets of a vertex per round
constexpr uint32_t kCoRecords = 8;     // records of a vertex per round
constexpr uint32_t kCoRow = 12;
constexpr uint32_t kCoStride = (kCoTets + kCoRecords) * kCoRow + 12;  // floats per vertex: neighbours' sums read other banks

// Contribution of cubature record `rec` of vertex v: w * projected gradient,
// the projected Hessian and the weight (0 for an empty record).
__device__ __forceinline__ float corotatedRecord(const Buffers& b, const DevParams& p, const float4* __restrict__ src,
                                                 uint32_t v, size_t rec, float* row) {
  const uint4 head = __ldg(&b.cubHead[2 * rec]);
  const float w = __uint_as_float(head.y);
  if (head.x == kEmptyTet || !(w > 0.0f)) return 0.0f;
  const uint4 info = b.vinfo[v];
  const float3 position = xyz(src[v]);
  const float4 pv = b.predicted[v];
  const float dWs = pv.w;
  const bool objActive = p.objectiveFlags != 0u;
  const M3 RsT = mtrans(loadFrame(b.vertexPack, v));
  const uint32_t t = head.x;
  const uint4 q = __ldg(&b.cubHead[2 * rec + 1]);
  const float4* U = b.cubBasis + 9ull * rec;
  M3 basis[4];
#pragma unroll
  for (int l = 0; l < 4; ++l) basis[l] = mm(mm(loadFrame(b.vertexPack, idxAt(q, l)), loadBlockVec(U, l)), RsT);
  const M3 R = loadRot(b.tetRot, t);
  const float* k = b.stiffness + 144ull * t;
  float3 disp[4], tg[4];
  corotatedDisplacement(b, src, q, R, disp);
  const M3 system = corotatedRecordSystem(k, R, disp, basis, tg);
  float3 pg = f3(0, 0, 0);
  M3 ih = mzero();
  uint32_t ss = 4;
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    const uint32_t qv = idxAt(q, l);
    if (qv == v) ss = l;
    const float4 pq = b.predicted[qv];
    const float3 xq = xyz(src[qv]);
    pg = pg + mtv(basis[l], tg[l] + pq.w * (xq - xyz(pq)));
    ih = ih + pq.w * mm(mtrans(basis[l]), basis[l]);
  }
  if (objActive) {
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      const uint32_t qv = idxAt(q, l);
      pg = pg + mtv(basis[l], distributedObjective(p, b, qv, xyz(src[qv]), b.vinfo[qv]));
    }
  }
  M3 ph = system + ih;
  if (p.objectiveFlags & 2u) {
    M3 oh = mzero();
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      const uint32_t qv = idxAt(q, l);
      const uint4 qi = b.vinfo[qv];
      const float kt = isPinned(qi) ? 0.0f : targetStiffness(p, b, qv) / float(qi.y > 1u ? qi.y : 1u);
      oh = oh + kt * mm(mtrans(basis[l]), basis[l]);
    }
    ph = ph + oh;
  }
  if (ss < 4) {
    const float3 own = ss == 0 ? tg[0] : ss == 1 ? tg[1] : ss == 2 ? tg[2] : tg[3];
    // The inertia share is rounded before it joins the record's gradient (it
    // belongs to the vertex, not to the record).
    const float3 away = position - xyz(pv);
    pg = pg - (own + f3(__fmul_rn(dWs, away.x), __fmul_rn(dWs, away.y), __fmul_rn(dWs, away.z)));
    if (objActive) {
      // The vertex's own share (it is not pinned) in one rounding, as the
      // one-thread-per-vertex form, which knew that, was contracted.
      const float3 og = objectiveGradient(p, b, v, position);
      const float share = 1.0f / float(info.y > 1u ? info.y : 1u);
      pg = f3(__fmaf_rn(-og.x, share, pg.x), __fmaf_rn(-og.y, share, pg.y), __fmaf_rn(-og.z, share, pg.z));
    }
    ph = ph - (mm(mm(R, stiffnessBlock(k, ss, ss)), mtrans(R)) + dWs * midentity());
    if (p.objectiveFlags & 2u)
      ph = ph - (targetStiffness(p, b, v) / float(info.y > 1u ? info.y : 1u)) * midentity();
  }
  pg = w * pg;
  row[0] = pg.x; row[1] = pg.y; row[2] = pg.z;
  row[3] = ph.c0.x; row[4] = ph.c0.y; row[5] = ph.c0.z;
  row[6] = ph.c1.x; row[7] = ph.c1.y; row[8] = ph.c1.z;
  row[9] = ph.c2.x; row[10] = ph.c2.y; row[11] = ph.c2.z;
  return w;
}

__device__ __forceinline__ void storeCoRow(float* dst, const float (&row)[kCoRow]) {
  float4* d = reinterpret_cast<float4*>(dst);
#pragma unroll
  for (uint32_t i = 0; i < kCoRow / 4; ++i)
    d[i] = make_float4(row[4 * i], row[4 * i + 1], row[4 * i + 2], row[4 * i + 3]);
}

__global__ void __launch_bounds__(kBlock, 2) corotatedSolveKernel(Buffers b, const DevParams* __restrict__ pp,
                                                               const float4* __restrict__ src, float4* tgt,
                                                               const uint32_t* __restrict__ list, uint32_t count,
                                                               uint32_t K) {
  __shared__ float4 rows4[kCoVertices * kCoStride / 4];
  __shared__ float weight[kCoVertices][kCoRecords];
  __shared__ uint32_t sVertex[kCoVertices], sStart[kCoVertices], sCount[kCoVertices];
  float* rows = reinterpret_cast<float*>(rows4);
  const uint32_t first = blockIdx.x * kCoVertices;
  uint32_t mine = 0;  // incident tets of this thread's vertex
  if (threadIdx.x < kCoVertices) {
    const uint32_t i = first + threadIdx.x;
    uint32_t v = kEmptyTet;
    if (i < count) {
      v = list ? list[i] : i;
      const uint4 info = b.vinfo[v];
      if (!pp[b.vertexScene[v]].active) {
        v = kEmptyTet;
      } else if (isPinned(info)) {
        const float4 rm = b.restMass[v];
        tgt[v] = make_float4(rm.x, rm.y, rm.z, 1.0f);
        b.finalUpdate[v] = 0.0f;
        v = kEmptyTet;
      } else {
        sStart[threadIdx.x] = info.x;
        mine = info.y;
      }
    }
    sVertex[threadIdx.x] = v;
    sCount[threadIdx.x] = mine;
  }
  __syncthreads();
  uint32_t most = 0;
  for (uint32_t g = 0; g < kCoVertices; ++g) most = max(most, sCount[g]);
  // This thread's component sum: component `comp` (gradient 0-2, Hessian
  // columns 3-11) of the block's vertex `sg`.
  const uint32_t sg = threadIdx.x / kCoRow, comp = threadIdx.x % kCoRow;
  const uint32_t sv = sg < kCoVertices ? sVertex[sg] : kEmptyTet;
  const bool sums = sv != kEmptyTet;
  float acc = 0.0f, low = 0.0f;  // gradient components: value and compensation
  auto gradientAdd = [&](float x) {
    float e;
    acc = twoSum(acc, x, &e);
    low = __fadd_rn(low, e);
  };
  auto component = [&](float3 a) { return comp == 0 ? a.x : comp == 1 ? a.y : a.z; };
  const bool diagonal = comp == 3 || comp == 7 || comp == 11;
  if (sums) {
    const DevParams& p = pp[b.vertexScene[sv]];
    const float4 rm = b.restMass[sv];
    const float inertia = rm.w * p.invDt2;
    if (comp < 3) {
      const float3 position = xyz(src[sv]);
      gradientAdd(component(inertia * (position - xyz(b.predicted[sv]))));
      if (p.objectiveFlags != 0u) gradientAdd(component(objectiveGradient(p, b, sv, position)));
    } else if (diagonal) {
      acc = inertia;
      if (p.objectiveFlags & 2u) acc = __fadd_rn(acc, targetStiffness(p, b, sv));
    }
  }
  auto record = [&](uint32_t g, uint32_t j, uint32_t s0) {
    const uint32_t v = sVertex[g];
    if (v == kEmptyTet) return;
    float row[kCoRow];
    const float w = corotatedRecord(b, pp[b.vertexScene[v]], src, v, static_cast<size_t>(v) * K + s0 + j, row);
    weight[g][j] = w;
    if (w > 0.0f) storeCoRow(rows + g * kCoStride + (kCoTets + j) * kCoRow, row);
  };
  auto tet = [&](uint32_t g, uint32_t j, uint32_t a0) {
    if (a0 + j >= sCount[g]) return;
    const uint32_t entry = __ldg(&b.adjacency[sStart[g] + a0 + j]);
    const uint32_t t = entry >> 2, slot = entry & 3u;
    const uint4 q = __ldg(reinterpret_cast<const uint4*>(b.tets) + 4ull * t + 3);
    const M3 R = loadRot(b.tetRot, t);
    const float* k = b.stiffness + 144ull * t;
    float3 disp[4];
    corotatedDisplacement(b, src, q, R, disp);
    const float3 tg = stiffnessTimes(stiffnessRow(k, slot), R, disp);
    const M3 h = mm(mm(R, stiffnessBlock(k, slot, slot)), mtrans(R));
    const float row[kCoRow] = {tg.x, tg.y, tg.z, h.c0.x, h.c0.y, h.c0.z, h.c1.x, h.c1.y, h.c1.z, h.c2.x, h.c2.y, h.c2.z};
    storeCoRow(rows + g * kCoStride + j * kCoRow, row);
  };
  // The first records (the long items) go first and beside the first tets;
  // their rows wait until the tets are added.
  const uint32_t firstRecords = min(kCoRecords, K);
  for (uint32_t item = threadIdx.x; item < kCoVertices * (firstRecords + kCoTets); item += kBlock) {
    if (item < kCoVertices * firstRecords) {
      record(item / firstRecords, item % firstRecords, 0);
    } else {
      const uint32_t i = item - kCoVertices * firstRecords;
      tet(i / kCoTets, i % kCoTets, 0);
    }
  }
  for (uint32_t a0 = 0; a0 == 0 || a0 < most; a0 += kCoTets) {
    if (a0 > 0)
      for (uint32_t item = threadIdx.x; item < kCoVertices * kCoTets; item += kBlock)
        tet(item / kCoTets, item % kCoTets, a0);
    __syncthreads();
    if (sums) {
      const uint32_t n = min(kCoTets, sCount[sg] > a0 ? sCount[sg] - a0 : 0u);
      const float* r = rows + sg * kCoStride + comp;
      if (comp < 3)
        for (uint32_t j = 0; j < n; ++j) gradientAdd(r[j * kCoRow]);
      else
        for (uint32_t j = 0; j < n; ++j) acc = __fadd_rn(acc, r[j * kCoRow]);
    }
    __syncthreads();
  }
  if (sums && (comp == 1 || comp == 7)) {
    const DevParams& p = pp[b.vertexScene[sv]];
    const float y = src[sv].y;
    if (p.floorStiffness > 0.0f && y < p.floorHeight) {
      if (comp == 1) gradientAdd(p.floorStiffness * (y - p.floorHeight));
      else acc = __fadd_rn(acc, p.floorStiffness);
    }
  }
  for (uint32_t s0 = 0; s0 < K; s0 += kCoRecords) {
    const uint32_t n = min(kCoRecords, K - s0);
    if (s0 > 0) {
      __syncthreads();
      for (uint32_t item = threadIdx.x; item < kCoVertices * n; item += kBlock) record(item / n, item % n, s0);
      __syncthreads();
    }
    if (sums) {
      const float* r = rows + sg * kCoStride + kCoTets * kCoRow + comp;
      for (uint32_t j = 0; j < n; ++j) {
        const float w = weight[sg][j];
        if (!(w > 0.0f)) continue;
        if (comp < 3) gradientAdd(r[j * kCoRow]);
        else acc = __fmaf_rn(w, r[j * kCoRow], acc);
      }
    }
  }
  if (sums) rows[sg * kCoStride + comp] = comp < 3 ? __fadd_rn(acc, low) : acc;
  __syncthreads();
  if (threadIdx.x >= kCoVertices || sVertex[threadIdx.x] == kEmptyTet) return;
  const uint32_t v = sVertex[threadIdx.x];
  const DevParams& p = pp[b.vertexScene[v]];
  const float* r = rows + threadIdx.x * kCoStride;
  const float3 gradient = f3(r[0], r[1], r[2]);
  const M3 hess = {f3(r[3], r[4], r[5]), f3(r[6], r[7], r[8]), f3(r[9], r[10], r[11])};
  const float3 position = xyz(src[v]);
  // Regularised Cholesky solve with the shift max(regularization * scale, 1e-9).
  const float ds = fmaxf(1.0f, fmaxf(fabsf(hess.c0.x), fmaxf(fabsf(hess.c1.y), fabsf(hess.c2.z))));
  const float shift = fmaxf(p.regularization * ds, 1.0e-9f);
  const float a00 = hess.c0.x + shift, a11 = hess.c1.y + shift, a22 = hess.c2.z + shift;
  const float a01 = 0.5f * (hess.c0.y + hess.c1.x);
  const float a02 = 0.5f * (hess.c0.z + hess.c2.x);
  const float a12 = 0.5f * (hess.c1.z + hess.c2.y);
  const float3 rhs = -gradient;
  const float l00 = sqrtf(fmaxf(a00, shift));
  const float l10 = a01 / l00, l20 = a02 / l00;
  const float l11 = sqrtf(fmaxf(a11 - l10 * l10, shift));
  const float l21 = (a12 - l20 * l10) / l11;
  const float l22 = sqrtf(fmaxf(a22 - l20 * l20 - l21 * l21, shift));
  const float y0 = rhs.x / l00, y1 = (rhs.y - l10 * y0) / l11, y2 = (rhs.z - l20 * y0 - l21 * y1) / l22;
  const float x2 = y2 / l22, x1 = (y1 - l21 * x2) / l11, x0 = (y0 - l10 * x1 - l20 * x2) / l00;
  float3 delta = f3(x0, x1, x2);
  // The fused form every step bound and update record has been taken with.
  auto squared = [](float3 d) { return __fmaf_rn(d.z, d.z, __fmaf_rn(d.x, d.x, __fmul_rn(d.y, d.y))); };
  const float sq = squared(delta);
  if (!(sq >= 0.0f && sq < 1.0e30f)) delta = f3(0, 0, 0);
  const float dls = squared(delta);
  if (p.maxStep > 0.0f && dls > p.maxStep * p.maxStep) delta = delta * (p.maxStep * (1.0f / sqrtf(dls)));
  const float3 np = position + delta;
  tgt[v] = make_float4(np.x, np.y, np.z, 1.0f);
  b.finalUpdate[v] = sqrtf(squared(delta));
}

__global__ void __launch_bounds__(kBlock) copyKernel(Buffers b, const DevParams* __restrict__ pp,
                                                     const float4* __restrict__ src, float4* __restrict__ dst,
                                                     uint32_t V) {
  const uint32_t i = blockIdx.x * kBlock + threadIdx.x;
  if (i < V && pp[b.vertexScene[i]].active) {
    const float4 s = src[i];
    dst[i] = make_float4(s.x, s.y, s.z, 1.0f);
  }
}

// ---------------------------------------------------------------------------
// IPC contact (jgs2-shader.ts:233-874, 2694-2917).

// Candidates listed this iteration: the broad phase's count with a contact
// surface, else the static total.  Candidate kernels stride over it.
__device__ __forceinline__ uint32_t contactListed(const Buffers& b) {
  return b.contactDynamic ? __ldcg(b.bpStatus) : b.contactCount;
}

__device__ __forceinline__ uint4 contactIndices(const Buffers& b, uint32_t c, uint32_t* type) {
  uint4 q = __ldg(&b.contactIdx[c]);
  *type = q.w >> 31;
  q.w &= 0x7fffffffu;
#if JGS2_BOUNDS_CHECKS
  // An out-of-range candidate vertex is recorded and read as vertex 0.
  if (!inBounds(q.x, b.vertexTotal, kSiteContactVertex)) q.x = 0;
  if (!inBounds(q.y, b.vertexTotal, kSiteContactVertex)) q.y = 0;
  if (!inBounds(q.z, b.vertexTotal, kSiteContactVertex)) q.z = 0;
  if (!inBounds(q.w, b.vertexTotal, kSiteContactVertex)) q.w = 0;
#endif
  return q;
}

__device__ __forceinline__ float3 posOverride(const float4* __restrict__ x, uint32_t q, uint32_t ov, float3 op) {
  return q == ov ? op : xyz(x[q]);
}

// ipcContactAtThreshold / ipcContactAtOverride (:594-668).
__device__ __forceinline__ ContactData contactAt(const Buffers& b, uint32_t c, const float4* __restrict__ x,
                                                 float threshold, uint32_t ov = 0xffffffffu,
                                                 float3 op = make_float3(0.f, 0.f, 0.f)) {
  uint32_t type;
  const uint4 q = contactIndices(b, c, &type);
  return ipcContactFromPositions(type, posOverride(x, q.x, ov, op), posOverride(x, q.y, ov, op),
                                 posOverride(x, q.z, ov, op), posOverride(x, q.w, ov, op), threshold);
}

// ipcContactRoundingReach (:505-509).
__device__ __forceinline__ float contactRoundingReach(const DevParams& p) {
  return fmaxf(fmaxf(p.sceneScale, p.ipcActivation), 1.0e-12f) * kUnitRoundoff * kPositionResolutionMultiplier;
}

// ipcCandidatePinnedMotionExceedsBound (:476-503).
__device__ __forceinline__ bool contactPinnedMotion(const Buffers& b, uint4 q, const float4* __restrict__ src,
                                                    float bound) {
  const uint32_t vs[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    if (!isPinned(b.vinfo[vs[l]])) continue;
    const float3 d = xyz(b.restMass[vs[l]]) - xyz(src[vs[l]]);
    const float len = length3(d);
    if (!finiteV(d) || !finiteS(len) || len > bound) return true;
  }
  return false;
}

// includeCandidate of buildActiveContactRows (:2742-2782): a candidate stays
// active unless its source cache is valid, beyond the reach a bounded step can
// cross, frictionless and free of unbounded pinned motion.  The decision
// depends on the candidate only, so every incident vertex agrees.
__device__ __forceinline__ bool contactIncluded(const Buffers& b, const DevParams& p, uint32_t c,
                                                const float4* __restrict__ src, float* near) {
  const float4* st = b.contactState + kContactStateWords * static_cast<size_t>(c);
  const ContactData k = ipcCached(st[kContactSource], st[kContactSourceWeights]);
  const bool friction = p.ipcFriction > 0.0f && st[kContactLagged].w > 0.0f;
  const bool bounded = p.maxStep > 0.0f;
  const float reach = p.ipcActivation + 2.0f * (fmaxf(p.maxStep, 0.0f) + contactRoundingReach(p));
  uint32_t type;
  const uint4 q = contactIndices(b, c, &type);
  const bool pinnedMotion = contactPinnedMotion(b, q, src, fmaxf(p.maxStep, 0.0f));
  *near = ipcNear(k.valid, k.distance, friction);
  return !k.valid || !bounded || k.distance <= reach || friction || pinnedMotion;
}

// Displacement since the frame start weighted by the lagged weights
// (ipcWeightedDisplacement, :686-708).
__device__ __forceinline__ float3 contactRelative(const Buffers& b, uint4 q, float4 w, const float4* __restrict__ x,
                                                  uint32_t ov, float3 op) {
  float3 r = w.x * (posOverride(x, q.x, ov, op) - xyz(b.old[q.x]));
  r = r + w.y * (posOverride(x, q.y, ov, op) - xyz(b.old[q.y]));
  r = r + w.z * (posOverride(x, q.z, ov, op) - xyz(b.old[q.z]));
  r = r + w.w * (posOverride(x, q.w, ov, op) - xyz(b.old[q.w]));
  return r;
}

// ipcCandidateEnergyFromContact (:710-741).
__device__ __forceinline__ float contactEnergy(const Buffers& b, const DevParams& p, uint32_t c, const ContactData& k,
                                               const float4* __restrict__ x, uint32_t ov, float3 op) {
  if (!k.valid || !(k.distance > p.ipcMinDistance)) return kF32Max;
  float e = p.ipcStiffness * ipcBarrier(k.distance, p.ipcActivation);
  const float4* st = b.contactState + kContactStateWords * static_cast<size_t>(c);
  const float4 lag = st[kContactLagged];
  if (p.ipcFriction > 0.0f && lag.w > 0.0f) {
    const float3 n = ipcSafeUnit(xyz(lag), k.normal);
    uint32_t type;
    const uint4 q = contactIndices(b, c, &type);
    const float3 rel = contactRelative(b, q, st[kContactLaggedWeights], x, ov, op);
    const float3 tang = rel - n * dot3(n, rel);
    e += p.dt * ipcFrictionDissipation(length3(tang) * p.invDt, p.ipcEpsilon, p.ipcFriction, lag.w);
  }
  return e;
}

// A lane's walk over a vertex's active candidates (`ids` at a, a + stride, ...):
// the ids and their near words are fetched four ahead, so that the walk does
// not wait for two dependent loads per candidate.
struct ContactBatch {
  uint32_t c0, c1, c2, c3;
  float d0, d1, d2, d3;
  uint32_t left = 0;
  __device__ __forceinline__ float next(const uint32_t* __restrict__ ids, const float* __restrict__ near, uint32_t a,
                                        uint32_t n, uint32_t stride, uint32_t* c) {
    if (left == 0) {
      c0 = ids[a];
      c1 = ids[min(a + stride, n - 1)];
      c2 = ids[min(a + 2 * stride, n - 1)];
      c3 = ids[min(a + 3 * stride, n - 1)];
      d0 = near[c0];
      d1 = near[c1];
      d2 = near[c2];
      d3 = near[c3];
      left = 4;
    }
    *c = c0;
    const float d = d0;
    c0 = c1; c1 = c2; c2 = c3;
    d0 = d1; d1 = d2; d2 = d3;
    --left;
    return d;
  }
};

// ipcLocalContribution (:788-869) over the vertex's active candidates
// [first, count) step `stride`: barrier gradient and PSD normal block, lagged
// friction gradient and tangential block.  `fresh` evaluates the contact at x
// (the coloured schedule), otherwise the cache at `slot` is used, whose
// distances are in `near`.
template <bool kHessian, class G>
__device__ __forceinline__ void contactLocal(const Buffers& b, const DevParams& p, uint32_t v,
                                             const float4* __restrict__ x, bool fresh, int slot,
                                             const float* __restrict__ near, uint32_t first, uint32_t stride, G& grad,
                                             S3& hess) {
  const uint2 range = b.contactRange[v];
  const uint32_t n = b.activeCount[v];
  ContactBatch batch;
  for (uint32_t a = first; a < n; a += stride) {
    uint32_t c;
    if (fresh) {
      c = b.activeIds[range.x + a];
    } else {
      const float d = batch.next(b.activeIds + range.x, near, a, n, stride, &c);
      if (!ipcNearValid(d) || !(ipcBarrierActive(fabsf(d), p.ipcActivation) || ipcNearFriction(d))) continue;
    }
    const float4* st = b.contactState + kContactStateWords * static_cast<size_t>(c);
    const ContactData k = fresh ? contactAt(b, c, x, p.ipcActivation) : ipcCached(st[slot], st[slot + 1]);
    if (!k.valid) continue;
    const bool barrier = ipcBarrierActive(k.distance, p.ipcActivation);
    const float4 lag = st[kContactLagged];
    const bool friction = p.ipcFriction > 0.0f && lag.w > 0.0f;
    if (!barrier && !friction) continue;
    uint32_t type;
    const uint4 q = contactIndices(b, c, &type);
    if (ipcWeightFor(q, make_float4(1.f, 1.f, 1.f, 1.f), v) == 0.0f) continue;
    const float w = ipcWeightFor(q, k.weights, v);
    if (w != 0.0f && barrier) {
      gadd(grad, ipcNormalGradientScalar(w, p.ipcStiffness, ipcBarrier1(k.distance, p.ipcActivation)) * k.normal);
      if (kHessian) {
        const float s = ipcPsdScalar(w, p.ipcStiffness, ipcBarrier2(k.distance, p.ipcActivation));
        saddOuter(hess, fmaxf(s, 0.0f), ipcSafeUnit(k.normal, f3(1, 0, 0)));
      }
    }
    const float4 lagW = st[kContactLaggedWeights];
    const float lw = ipcWeightFor(q, lagW, v);
    if (friction && lw != 0.0f) {
      const float3 nrm = ipcSafeUnit(xyz(lag), k.normal);
      const float3 rel = contactRelative(b, q, lagW, x, 0xffffffffu, f3(0, 0, 0));
      const float3 tang = rel - nrm * dot3(nrm, rel);
      const float slip = length3(tang);
      const float scale = p.ipcFriction * lag.w;
      const float3 dir = slip > 1.0e-12f ? tang * (1.0f / slip) : f3(0, 0, 0);
      const float f1 = ipcFrictionF1(slip * p.invDt, p.ipcEpsilon);
      gadd(grad, (lw * scale * f1) * dir);
      if (kHessian) {
        float curvature = 2.0f * scale / fmaxf(p.ipcEpsilon * p.dt, 1.0e-12f);
        if (slip > 1.0e-12f) curvature = scale * f1 / slip;
        const float c2 = lw * lw * fmaxf(curvature, 0.0f);
        saddDiag(hess, c2);
        saddOuter(hess, -c2, ipcSafeUnit(nrm, f3(1, 0, 0)));
      }
    }
  }
}

// JGS2_CONTACT_MIN_BLOCKS: blocks per SM the register budgets of the
// per-candidate contact kernels (lag, safe step, validation, broad-phase
// initialisation) must allow (0: the compiler's choice).
#ifndef JGS2_CONTACT_MIN_BLOCKS
#define JGS2_CONTACT_MIN_BLOCKS 0
#endif
#if JGS2_CONTACT_MIN_BLOCKS > 0
#define JGS2_CONTACT_BOUNDS __launch_bounds__(kBlock, JGS2_CONTACT_MIN_BLOCKS)
#else
#define JGS2_CONTACT_BOUNDS __launch_bounds__(kBlock)
#endif

// lagContact (:2712-2740): source cache and lagged normal force at the
// accepted pose, once per frame.
__global__ void JGS2_CONTACT_BOUNDS contactLagKernel(Buffers b, const DevParams* __restrict__ pp) {
  const uint32_t c = blockIdx.x * kBlock + threadIdx.x;
  if (c >= b.contactCount) return;
  const uint32_t scene = b.contactScene[c];
  const DevParams& p = pp[scene];
  if (!p.active || !p.ipc) return;
  const ContactData k = contactAt(b, c, b.pos[0], p.ipcActivation + contactRoundingReach(p));
  float4* st = b.contactState + kContactStateWords * static_cast<size_t>(c);
  ipcStoreCached(st, kContactSource, k);
  float4 force = make_float4(0, 0, 0, 0), w = make_float4(0, 0, 0, 0);
  if (k.valid && k.distance > p.ipcMinDistance) {
    const float f = fmaxf(0.0f, -p.ipcStiffness * ipcBarrier1(k.distance, p.ipcActivation));
    if (finiteS(f)) {
      force = make_float4(k.normal.x, k.normal.y, k.normal.z, f);
      w = k.weights;
    }
  }
  st[kContactLagged] = force;
  st[kContactLaggedWeights] = w;
  if (c == b.scenes[scene].kOff) b.frames[scene].contactAlpha = 1.0f;
}

// buildActiveContactRows (:2742-2782) in two passes: the candidate's
// inclusion (a property of the candidate alone), with the reset of the
// iteration's safe-step reductions...
__global__ void __launch_bounds__(kBlock) contactFlagKernel(Buffers b, const DevParams* __restrict__ pp,
                                                            const float4* __restrict__ src) {
  const uint32_t c = blockIdx.x * kBlock + threadIdx.x;
  if (c >= b.contactCount) return;
  const uint32_t scene = b.contactScene[c];
  const DevParams& p = pp[scene];
  if (!p.active || !p.ipc) return;
  if (c == b.scenes[scene].kOff) {
    FrameState* fs = &b.frames[scene];
    fs->stepAlphaBits = __float_as_uint(1.0f);
    fs->stepValid = 1u;
    fs->checkAlphaBits = __float_as_uint(1.0f);
    fs->checkValid = 1u;
  }
  float near;
  b.contactFlag[c] = contactIncluded(b, p, c, src, &near) ? 1u : 0u;
  b.contactNear[c] = near;
}

// ...then, one warp per vertex, the ordered compaction of its included
// incident candidates into its active row.
__global__ void __launch_bounds__(kBlock) contactRowsKernel(Buffers b, const DevParams* __restrict__ pp,
                                                            uint32_t V) {
  const uint32_t v = blockIdx.x * (kBlock / 32) + threadIdx.x / 32;
  const uint32_t lane = threadIdx.x & 31u;
  if (v >= V) return;  // uniform across the warp
  const DevParams& p = pp[b.vertexScene[v]];
  if (!p.active || !p.ipc) return;
  const uint2 r = b.contactRange[v];
  uint32_t n = 0;
  // Eight rounds of 32 candidates in flight: a vertex of the reference's trough
  // has about 1 400, and one round at a time (an index, then its flag) took
  // 39 us.
  constexpr uint32_t kAhead = 8;
  for (uint32_t k0 = 0; k0 < r.y; k0 += 32 * kAhead) {
    uint32_t c[kAhead];
    bool keep[kAhead];
#pragma unroll
    for (uint32_t j = 0; j < kAhead; ++j) {
      const uint32_t k = k0 + 32 * j + lane;
      c[j] = k < r.y ? b.contactIds[r.x + k] : 0u;
    }
#pragma unroll
    for (uint32_t j = 0; j < kAhead; ++j) keep[j] = k0 + 32 * j + lane < r.y && b.contactFlag[c[j]] != 0u;
#pragma unroll
    for (uint32_t j = 0; j < kAhead; ++j) {
      const unsigned ballot = __ballot_sync(0xffffffffu, keep[j]);
      if (keep[j]) b.activeIds[r.x + n + __popc(ballot & ((1u << lane) - 1u))] = c[j];
      n += __popc(ballot);
    }
  }
  if (lane == 0) b.activeCount[v] = n;
}

// The IPC part of convergenceGradient's contact component (:4086-4088) at
// the accepted pose, one warp per vertex, from the contacts the promotion
// pass makes the next source cache.
__global__ void __launch_bounds__(kBlock) contactGradientKernel(Buffers b, const DevParams* __restrict__ pp,
                                                                const float4* __restrict__ src,
                                                                const float4* __restrict__ tgt, uint32_t V) {
  const uint32_t v = blockIdx.x * (kBlock / 32) + threadIdx.x / 32;
  const uint32_t lane = threadIdx.x & 31u;
  if (v >= V) return;  // uniform across the warp
  const uint32_t scene = b.vertexScene[v];
  const DevParams& p = pp[scene];
  const FrameState* fs = &b.frames[scene];
  if (!p.active || !p.ipc || latched(p, fs)) return;
  if (isPinned(b.vinfo[v])) return;
  const bool accepted = fs->control[1].x == 1.0f;
  const float alpha = fs->contactAlpha;
  const int slot = (accepted && finiteS(alpha) && alpha > 0.0f) ? kContactTarget : kContactSource;
  float3 g = f3(0, 0, 0);
  S3 unused = szero();
  contactLocal<false>(b, p, v, accepted ? tgt : src, false, slot,
                      slot == kContactTarget ? b.contactTargetNear : b.contactNear, lane, 32u, g, unused);
  g.x = groupSum<32>(g.x, 0xffffffffu);
  g.y = groupSum<32>(g.y, 0xffffffffu);
  g.z = groupSum<32>(g.z, 0xffffffffu);
  if (lane == 0) b.contactGrad[v] = make_float4(g.x, g.y, g.z, 0.0f);
}

__device__ __forceinline__ uint32_t alphaBits(float a) { return a > 0.0f ? __float_as_uint(a) : 0u; }

// Each vertex's step length this iteration, or -1 when the step is not finite
// (the candidate is then invalid whatever the other lengths are).
__global__ void __launch_bounds__(kBlock) contactMoveKernel(Buffers b, const float4* __restrict__ src,
                                                            const float4* __restrict__ tgt, uint32_t V) {
  const uint32_t v = blockIdx.x * kBlock + threadIdx.x;
  if (v >= V) return;
  const float3 d = xyz(tgt[v]) - xyz(src[v]);
  b.contactMove[v] = finiteV(d) ? length3(d) : -1.0f;
}

// candidateContactStep of one candidate.  kMoves: the step lengths come from
// contactMoveKernel, four 4-byte gathers instead of eight of 16 bytes.
template <bool kMoves>
__device__ __forceinline__ void contactStepOne(const Buffers& b, const DevParams* __restrict__ pp,
                                               const float4* __restrict__ src, const float4* __restrict__ tgt,
                                               uint32_t c) {
  const uint32_t scene = b.contactScene[c];
  const DevParams& p = pp[scene];
  if (!p.active || !p.ipc) return;
  FrameState* fs = &b.frames[scene];
  if (latched(p, fs)) return;  // alpha one, valid: the reduction's identity
  uint32_t type;
  const uint4 q = contactIndices(b, c, &type);
  float l0, l1, l2, l3;
  bool trialValid;
  if (kMoves) {
    const float m0 = b.contactMove[q.x], m1 = b.contactMove[q.y], m2 = b.contactMove[q.z], m3 = b.contactMove[q.w];
    l0 = m0; l1 = m1; l2 = m2; l3 = m3;
    trialValid = m0 >= 0.0f && m1 >= 0.0f && m2 >= 0.0f && m3 >= 0.0f;
  } else {
    const float3 d0 = xyz(tgt[q.x]) - xyz(src[q.x]), d1 = xyz(tgt[q.y]) - xyz(src[q.y]);
    const float3 d2 = xyz(tgt[q.z]) - xyz(src[q.z]), d3 = xyz(tgt[q.w]) - xyz(src[q.w]);
    l0 = length3(d0); l1 = length3(d1); l2 = length3(d2); l3 = length3(d3);
    trialValid = finiteV(d0) && finiteV(d1) && finiteV(d2) && finiteV(d3);
  }
  const float L = type == kIpcVertexTriangle ? l0 + fmaxf(l1, fmaxf(l2, l3)) : fmaxf(l0, l1) + fmaxf(l2, l3);
  const float near = b.contactNear[c];
  bool sourceValid = ipcNearValid(near);
  float distance = fabsf(near);
  bool fullStepSafe = sourceValid && finiteS(L) && distance - L > p.ipcMinDistance;
  if (!fullStepSafe) {
    const ContactData source = contactAt(b, c, src, kF32Max);
    sourceValid = source.valid;
    distance = source.distance;
    fullStepSafe = sourceValid && finiteS(L) && distance - L > p.ipcMinDistance;
  }
  const bool valid = sourceValid && trialValid && distance > p.ipcMinDistance && finiteS(L);
  float alpha = 0.0f;
  if (valid) alpha = fullStepSafe ? 1.0f : ipcSafeStepCap(distance, p.ipcMinDistance, L, p.ipcSafety);
  if (valid && finiteS(alpha)) {
    if (alpha < 1.0f) atomicMin(&fs->stepAlphaBits, alphaBits(alpha));
  } else {
    atomicMin(&fs->stepAlphaBits, 0u);
    atomicAnd(&fs->stepValid, 0u);
  }
}

// candidateContactStep (:2784-2847) with the min / all-valid reduction of
// reduceContactStep folded in as order-free atomics.
template <bool kMoves>
__global__ void JGS2_CONTACT_BOUNDS contactStepKernel(Buffers b, const DevParams* __restrict__ pp,
                                                            const float4* __restrict__ src,
                                                            const float4* __restrict__ tgt) {
  const uint32_t n = contactListed(b);
  for (uint32_t c = blockIdx.x * kBlock + threadIdx.x; c < n; c += gridDim.x * kBlock)
    contactStepOne<kMoves>(b, pp, src, tgt, c);
}

// applyContactStep (:2909-2917): candidate = source + alpha (candidate -
// source) with the safe-step alpha, or after validation with 1 (kept) or 0
// (restored); the validated alpha becomes the iteration's contact alpha.
__global__ void __launch_bounds__(kBlock) contactApplyKernel(Buffers b, const DevParams* __restrict__ pp,
                                                             const float4* __restrict__ src, float4* tgt,
                                                             uint32_t V, int validated) {
  const uint32_t v = blockIdx.x * kBlock + threadIdx.x;
  if (v >= V) return;
  const uint32_t scene = b.vertexScene[v];
  const DevParams& p = pp[scene];
  if (!p.active || !p.ipc) return;
  FrameState* fs = &b.frames[scene];
  const uint32_t bits = validated ? fs->checkAlphaBits : fs->stepAlphaBits;
  const uint32_t ok = validated ? fs->checkValid : fs->stepValid;
  const float alpha = ok ? clamp01f(__uint_as_float(bits)) : 0.0f;
  if (validated && v == b.scenes[scene].vOff) fs->contactAlpha = alpha;
  if (latched(p, fs)) return;
  const float3 s = xyz(src[v]);
  const float3 t = s + alpha * (xyz(tgt[v]) - s);
  tgt[v] = make_float4(t.x, t.y, t.z, 1.0f);
}

// validateContactStep (:2849-2868): exact contacts of the scaled candidate
// (the target cache) and the all-valid reduction.
__global__ void JGS2_CONTACT_BOUNDS contactValidateKernel(Buffers b, const DevParams* __restrict__ pp,
                                                                const float4* __restrict__ tgt) {
  const uint32_t n = contactListed(b);
  for (uint32_t c = blockIdx.x * kBlock + threadIdx.x; c < n; c += gridDim.x * kBlock) {
    const uint32_t scene = b.contactScene[c];
    const DevParams& p = pp[scene];
    if (!p.active || !p.ipc) continue;
    FrameState* fs = &b.frames[scene];
    const ContactData k = contactAt(b, c, tgt, p.ipcActivation + contactRoundingReach(p));
    float4* st = b.contactState + kContactStateWords * static_cast<size_t>(c);
    ipcStoreCached(st, kContactTarget, k);
    const ContactData stored = ipcCached(st[kContactTarget], st[kContactTargetWeights]);
    b.contactTargetNear[c] = ipcNear(stored.valid, stored.distance, ipcNearFriction(b.contactNear[c]));
    const bool valid = k.valid && finiteS(k.distance) && k.distance > p.ipcMinDistance;
    if (!valid) {
      atomicMin(&fs->checkAlphaBits, 0u);
      atomicAnd(&fs->checkValid, 0u);
    }
  }
}

// Closest features of caller-given pairs (a diagnostic, not part of the
// step): the device routine every contact pass uses, f32 with the FP64 run
// for near-degenerate pairs; 9 floats per pair out (distance, normal,
// weights, valid) and whether the FP64 run was taken.
__global__ void __launch_bounds__(kBlock) contactFeatureKernel(const float* __restrict__ points,
                                                               const uint32_t* __restrict__ types, uint32_t n,
                                                               float* __restrict__ out, uint32_t* __restrict__ wide) {
  const uint32_t i = blockIdx.x * kBlock + threadIdx.x;
  if (i >= n) return;
  const float* x = points + 12ull * i;
  const float3 p0 = f3(x[0], x[1], x[2]), p1 = f3(x[3], x[4], x[5]);
  const float3 p2 = f3(x[6], x[7], x[8]), p3 = f3(x[9], x[10], x[11]);
  bool w = false;
  const ContactData k = types[i] == kIpcVertexTriangle ? ipcPointTriangle(p0, p1, p2, p3, &w)
                                                       : ipcEdgeEdge(p0, p1, p2, p3, &w);
  float* o = out + 9ull * i;
  o[0] = k.distance;
  o[1] = k.normal.x; o[2] = k.normal.y; o[3] = k.normal.z;
  o[4] = k.weights.x; o[5] = k.weights.y; o[6] = k.weights.z; o[7] = k.weights.w;
  o[8] = k.valid ? 1.0f : 0.0f;
  wide[i] = w ? 1u : 0u;
}

// promoteAcceptedContactCache (:2694-2710).
__global__ void __launch_bounds__(kBlock) contactPromoteKernel(Buffers b, const DevParams* __restrict__ pp) {
  const uint32_t n = contactListed(b);
  for (uint32_t c = blockIdx.x * kBlock + threadIdx.x; c < n; c += gridDim.x * kBlock) {
    const uint32_t scene = b.contactScene[c];
    const DevParams& p = pp[scene];
    if (!p.active || !p.ipc) continue;
    const FrameState* fs = &b.frames[scene];
    const float alpha = fs->contactAlpha;
    if (fs->control[1].x == 1.0f && finiteS(alpha) && alpha > 0.0f) {
      float4* st = b.contactState + kContactStateWords * static_cast<size_t>(c);
      st[kContactSource] = st[kContactTarget];
      st[kContactSourceWeights] = st[kContactTargetWeights];
      b.contactNear[c] = b.contactTargetNear[c];
    }
  }
}

// ---------------------------------------------------------------------------
// IPC broad phase over the static candidate superset (contact surfaces).
//
// The superset (buildStaticIpcContactCandidates, ipc-contact.ts:591-665) is
// never listed.  Every iteration one warp per row (a vertex against its
// scene's surface triangles, or a surface edge against the later edges)
// walks the row's columns in canonical order, 32-primitive chunk boxes
// first, and lists the pairs whose boxes, each widened by the largest motion
// its vertices can make this iteration, are not separated by more than the
// activation distance plus the rounding reach; pairs of the previous list
// that carry lagged friction stay listed for the frame.  A pair left out is
// farther than that from every pose the iteration can produce, so the
// reference's passes give it no active row, a full safe step, a valid check
// and no energy: it does not act.  A listed pair's state is carried from the
// previous list (the promoted source cache, the lagged friction) or formed
// from the source pose as lagContact does.  The per-vertex active rows come
// from a stable radix sort of the active candidates' vertex entries, so each
// row keeps ascending candidate order, as the static rows do.

constexpr uint32_t kBpChunk = 32;
constexpr uint32_t kBpClosedMax = 64;  // closed one-ring vertices a row keeps in shared memory
constexpr float kBpInf = __builtin_huge_valf();

struct BpBox {
  float3 lo, hi;
  float m;  // largest motion of the primitive's vertices this iteration
};

// A vertex's largest displacement in one iteration: maxStep for a free
// vertex (the line search caps each local step at maxStep, :3322-3445) and
// the snap to rest for a pinned one, widened by a relative 2^-12 and 16 ulps
// of the coordinates for the rounding of the committed positions.
__device__ __forceinline__ float bpMotion(const Buffers& b, const DevParams& p, uint32_t v, float3 x) {
  float m = fmaxf(p.maxStep, 0.0f);
  if (isPinned(b.vinfo[v])) m = fmaxf(m, length3(xyz(b.restMass[v]) - x));
  const float ax = fmaxf(fabsf(x.x), fmaxf(fabsf(x.y), fabsf(x.z)));
  const float r = m * (1.0f + 0x1p-12f) + ax * 0x1p-19f;
  return finiteS(r) ? r : kBpInf;
}

__device__ __forceinline__ BpBox bpEmpty() { return {f3(kBpInf, kBpInf, kBpInf), f3(-kBpInf, -kBpInf, -kBpInf), 0.0f}; }
__device__ __forceinline__ BpBox bpEverything() {
  return {f3(-kBpInf, -kBpInf, -kBpInf), f3(kBpInf, kBpInf, kBpInf), kBpInf};
}

// Bounds and largest motion of a primitive at x; non-finite data widens it
// to everything (such a pair is always listed, as the static path keeps it).
template <int N>
__device__ __forceinline__ BpBox bpPrimitive(const Buffers& b, const DevParams& p, const float4* __restrict__ x,
                                             const uint32_t (&vs)[N]) {
  BpBox q = bpEmpty();
  bool ok = true;
#pragma unroll
  for (int l = 0; l < N; ++l) {
    const float3 y = xyz(x[vs[l]]);
    ok = ok && finiteV(y);
    q.lo = fmin3(q.lo, y);
    q.hi = fmax3(q.hi, y);
    q.m = fmaxf(q.m, bpMotion(b, p, vs[l], y));
  }
  return (ok && finiteS(q.m)) ? q : bpEverything();
}

__device__ __forceinline__ void bpStore(float4* boxes, uint32_t i, const BpBox& q) {
  boxes[2ull * i] = make_float4(q.lo.x, q.lo.y, q.lo.z, q.m);
  boxes[2ull * i + 1] = make_float4(q.hi.x, q.hi.y, q.hi.z, 0.0f);
}
__device__ __forceinline__ BpBox bpLoad(const float4* __restrict__ boxes, uint32_t i) {
  const float4 a = boxes[2ull * i], c = boxes[2ull * i + 1];
  return {f3(a.x, a.y, a.z), f3(c.x, c.y, c.z), a.w};
}

// Separated by more than `reach` once both boxes are widened by their
// motions: the per-axis gaps less the motions, as a Euclidean length.  Each
// step is monotone in the boxes, so a chunk box that contains a primitive's
// box (and its motion) separates no more than the primitive's does.
__device__ __forceinline__ bool bpSeparated(const BpBox& a, const BpBox& c, float reach) {
  const float m = a.m + c.m;
  const float3 g = fmax3(fmax3(c.lo - a.hi, a.lo - c.hi), f3(0, 0, 0));
  const float3 h = fmax3(g - f3(m, m, m), f3(0, 0, 0));
  return dot3(h, h) > reach * reach;
}

// The activation distance and twice the rounding reach
// (ipcActiveContactReach less its step terms, which the motions carry),
// widened by 2^-10.
__device__ __forceinline__ float bpReach(const DevParams& p) {
  return (p.ipcActivation + 2.0f * contactRoundingReach(p)) * (1.0f + 0x1p-10f);
}

// closed(a, v) of the enumeration: a == v or v in a's surface one-ring.
__device__ __forceinline__ bool bpClosed(const Buffers& b, uint32_t a, uint32_t v) {
  if (a == v) return true;
  const uint2 r = b.bpRing[a];
  for (uint32_t i = 0; i < r.y; ++i)
    if (b.bpRingIds[r.x + i] == v) return true;
  return false;
}

// The superset leaves out a vertex and a triangle of its closed one-ring,
// and two edges with an endpoint of one in the other's closed one-rings.
__device__ __forceinline__ bool bpPairClosed(const Buffers& b, bool edgeRow, const uint32_t (&rv)[2], uint32_t col) {
  if (!edgeRow) {
    const uint4 t = b.bpTris[col];
    return bpClosed(b, rv[0], t.x) || bpClosed(b, rv[0], t.y) || bpClosed(b, rv[0], t.z);
  }
  const uint2 e = b.bpEdges[col];
  return bpClosed(b, rv[0], e.x) || bpClosed(b, rv[0], e.y) || bpClosed(b, rv[1], e.x) || bpClosed(b, rv[1], e.y);
}

// Primitive and chunk boxes at the iteration's source pose (a warp's 32
// primitives form one chunk), and the reset of every vertex's active row.
__global__ void __launch_bounds__(kBlock) bpBoxesKernel(Buffers b, const DevParams* __restrict__ pp,
                                                        const float4* __restrict__ src, uint32_t triBlocks,
                                                        uint32_t edgeBlocks, uint32_t V) {
  const uint32_t blk = blockIdx.x;
  if (blk < triBlocks + edgeBlocks) {
    const bool edges = blk >= triBlocks;
    const uint32_t i = (edges ? blk - triBlocks : blk) * kBlock + threadIdx.x;
    const uint32_t n = edges ? b.bpEdgeTotal : b.bpTriTotal;
    BpBox q = bpEmpty();
    if (i < n) {
      if (edges) {
        const uint2 e = b.bpEdges[i];
        const uint32_t vs[2] = {e.x, e.y};
        q = bpPrimitive(b, pp[b.vertexScene[e.x]], src, vs);
        bpStore(b.bpEdgeBox, i, q);
      } else {
        const uint4 t = b.bpTris[i];
        const uint32_t vs[3] = {t.x, t.y, t.z};
        q = bpPrimitive(b, pp[t.w], src, vs);
        bpStore(b.bpTriBox, i, q);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      q.lo.x = fminf(q.lo.x, __shfl_xor_sync(0xffffffffu, q.lo.x, o));
      q.lo.y = fminf(q.lo.y, __shfl_xor_sync(0xffffffffu, q.lo.y, o));
      q.lo.z = fminf(q.lo.z, __shfl_xor_sync(0xffffffffu, q.lo.z, o));
      q.hi.x = fmaxf(q.hi.x, __shfl_xor_sync(0xffffffffu, q.hi.x, o));
      q.hi.y = fmaxf(q.hi.y, __shfl_xor_sync(0xffffffffu, q.hi.y, o));
      q.hi.z = fmaxf(q.hi.z, __shfl_xor_sync(0xffffffffu, q.hi.z, o));
      q.m = fmaxf(q.m, __shfl_xor_sync(0xffffffffu, q.m, o));
    }
    if ((threadIdx.x & 31u) == 0u && i < n) bpStore(edges ? b.bpEdgeChunk : b.bpTriChunk, i / kBpChunk, q);
    return;
  }
  const uint32_t v = (blk - triBlocks - edgeBlocks) * kBlock + threadIdx.x;
  if (v >= V) return;
  b.activeCount[v] = 0u;
  // ipcCandidatePinnedMotionExceedsBound per vertex (contactPinnedMotion).
  uint32_t move = 0u;
  if (isPinned(b.vinfo[v])) {
    const DevParams& p = pp[b.vertexScene[v]];
    const float3 d = xyz(b.restMass[v]) - xyz(src[v]);
    const float len = length3(d);
    move = (!finiteV(d) || !finiteS(len) || len > fmaxf(p.maxStep, 0.0f)) ? 1u : 0u;
  }
  b.bpPinnedMove[v] = move;
}

// Superchunk boxes: one warp per 32 chunks (the union of their boxes).
__global__ void __launch_bounds__(kBlock) bpSuperKernel(Buffers b, uint32_t triSupers, uint32_t edgeSupers) {
  const uint32_t w = blockIdx.x * (kBlock / 32) + threadIdx.x / 32, lane = threadIdx.x & 31u;
  if (w >= triSupers + edgeSupers) return;  // uniform across the warp
  const bool edges = w >= triSupers;
  const uint32_t sc = edges ? w - triSupers : w;
  const uint32_t chunks = ((edges ? b.bpEdgeTotal : b.bpTriTotal) + kBpChunk - 1) / kBpChunk;
  const uint32_t chunk = sc * kBpChunk + lane;
  BpBox q = chunk < chunks ? bpLoad(edges ? b.bpEdgeChunk : b.bpTriChunk, chunk) : bpEmpty();
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    q.lo.x = fminf(q.lo.x, __shfl_xor_sync(0xffffffffu, q.lo.x, o));
    q.lo.y = fminf(q.lo.y, __shfl_xor_sync(0xffffffffu, q.lo.y, o));
    q.lo.z = fminf(q.lo.z, __shfl_xor_sync(0xffffffffu, q.lo.z, o));
    q.hi.x = fmaxf(q.hi.x, __shfl_xor_sync(0xffffffffu, q.hi.x, o));
    q.hi.y = fmaxf(q.hi.y, __shfl_xor_sync(0xffffffffu, q.hi.y, o));
    q.hi.z = fmaxf(q.hi.z, __shfl_xor_sync(0xffffffffu, q.hi.z, o));
    q.m = fmaxf(q.m, __shfl_xor_sync(0xffffffffu, q.m, o));
  }
  if (lane == 0) bpStore(edges ? b.bpEdgeSuper : b.bpTriSuper, sc, q);
}

// A listed pair's state: carried from the previous list (its entry
// `bpPrev`), else the source contact and, at the frame's first iteration, its
// lagged force as lagContact (:2712-2740) forms them; its activity
// (contactIncluded) and its four sort entries (vertex, candidate), whose key
// is the sentinel when the pair is inactive.  One thread per candidate.
__global__ void JGS2_CONTACT_BOUNDS bpInitKernel(Buffers b, const DevParams* __restrict__ pp,
                                                       const float4* __restrict__ src, int first) {
  const uint32_t n = __ldcg(b.bpStatus);
  for (uint32_t c = blockIdx.x * kBlock + threadIdx.x; c < n; c += gridDim.x * kBlock) {
    const DevParams& p = pp[b.contactScene[c]];
    uint32_t type;
    const uint4 q = contactIndices(b, c, &type);
    float4* st = b.contactState + kContactStateWords * static_cast<size_t>(c);
    float4 lagF = make_float4(0, 0, 0, 0), lagW = make_float4(0, 0, 0, 0);
    const uint32_t prev = first ? 0xffffffffu : b.bpPrev[c];
    float4 s0, s1;
    if (prev != 0xffffffffu) {
      // promoteAcceptedContactCache (:2694-2710) of the previous iteration: the
      // target contacts of an accepted pose become the source cache.
      const FrameState* fs = &b.frames[b.contactScene[c]];
      const float alpha = fs->contactAlpha;
      const int slot = fs->control[1].x == 1.0f && finiteS(alpha) && alpha > 0.0f ? kContactTarget : kContactSource;
      const float4* ps = b.bpPrevState + kContactStateWords * static_cast<size_t>(prev);
      s0 = ps[slot];
      s1 = ps[slot + 1];
      lagF = ps[kContactLagged];
      lagW = ps[kContactLaggedWeights];
      st[kContactSource] = s0;
      st[kContactSourceWeights] = s1;
    } else {
      const ContactData k = ipcContactFromPositions(type, xyz(src[q.x]), xyz(src[q.y]), xyz(src[q.z]), xyz(src[q.w]),
                                                    p.ipcActivation + contactRoundingReach(p));
      ipcStoreCached(st, kContactSource, k);
      s0 = st[kContactSource];
      s1 = st[kContactSourceWeights];
      if (first && k.valid && k.distance > p.ipcMinDistance) {
        const float f = fmaxf(0.0f, -p.ipcStiffness * ipcBarrier1(k.distance, p.ipcActivation));
        if (finiteS(f)) {
          lagF = make_float4(k.normal.x, k.normal.y, k.normal.z, f);
          lagW = k.weights;
        }
      }
    }
    st[kContactLagged] = lagF;
    st[kContactLaggedWeights] = lagW;
    // contactIncluded on the state just written.
    const ContactData k = ipcCached(s0, s1);
    const bool friction = p.ipcFriction > 0.0f && lagF.w > 0.0f;
    b.contactNear[c] = ipcNear(k.valid, k.distance, friction);
    const bool bounded = p.maxStep > 0.0f;
    const float reach = p.ipcActivation + 2.0f * (fmaxf(p.maxStep, 0.0f) + contactRoundingReach(p));
    const bool pinnedMove =
        (b.bpPinnedMove[q.x] | b.bpPinnedMove[q.y] | b.bpPinnedMove[q.z] | b.bpPinnedMove[q.w]) != 0u;
    const bool active = !k.valid || !bounded || k.distance <= reach || friction || pinnedMove;
    b.contactFlag[c] = active ? 1u : 0u;
    const uint32_t key = b.bpSentinel;
    reinterpret_cast<uint4*>(b.bpKeys[0])[c] =
        active ? make_uint4(q.x, q.y, q.z, q.w) : make_uint4(key, key, key, key);
  }
}

// One warp per row: the row's pairs in column order, counted (kWrite false,
// into bpRowOff[row]) or placed at the row's offset with their previous
// entry (kWrite true).  The count keeps a row's first kBpRowHits hit chunks with
// their masks, from which the write pass places the pairs without testing any
// box; a row with more walks them again.  The columns are walked 32 superchunks (of 32 chunks
// of 32 primitives) at a time, then 32 chunks, then 32 primitives, each
// level only inside the boxes the row's box does not clear.
template <bool kWrite>
__global__ void __launch_bounds__(kBlock) bpRowsKernel(Buffers b, const DevParams* __restrict__ pp,
                                                       const float4* __restrict__ src, int first) {
  __shared__ uint32_t carried[kBlock / 32][32];
  __shared__ uint32_t closedSet[kBlock / 32][kBpClosedMax];
  const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x & 31u;
  const uint32_t r = blockIdx.x * (kBlock / 32) + warp;
  if (r >= b.bpRowTotal) return;                   // uniform across the warp
  if (kWrite && __ldcg(&b.bpStatus[3])) return;   // over capacity: nothing listed this iteration
  const uint4 row = b.bpRows[r];
  const uint32_t scene = row.y & 0x7fffffffu;
  const bool edgeRow = (row.y >> 31) != 0u;
  const DevParams& p = pp[scene];
  uint32_t count = 0;
  if (p.active && p.ipc && row.z < row.w) {
    uint32_t rv[2];
    if (edgeRow) {
      const uint2 e = b.bpEdges[row.x];
      rv[0] = e.x;
      rv[1] = e.y;
    } else {
      rv[0] = rv[1] = row.x;
    }
    const uint32_t base = kWrite ? b.bpRowOff[r] : 0u;
    uint32_t pc = 0, pe = 0;  // this row's entries of the previous list
    if (!first) {
      pc = b.bpPrevRowOff[r];
      pe = b.bpPrevRowOff[r + 1];
    }
    // Carry cursor: the previous entries [qc, qc + 64), in w0 and w1.
    uint32_t qc = pc;
    uint32_t w0 = 0xffffffffu, w1 = 0xffffffffu;
    if (kWrite && !first) {
      if (pc + lane < pe) w0 = b.bpPrevCols[pc + lane];
      if (pc + 32 + lane < pe) w1 = b.bpPrevCols[pc + 32 + lane];
    }
    // Places the hits `m` of a chunk (this lane's column `col`, hit or not).
    auto place = [&](uint32_t chunk, unsigned m) {
      const uint32_t col = chunk * kBpChunk + lane;
      const bool hit = (m >> lane) & 1u;
      // The previous list's entries of this chunk (sorted, at most 32):
      // a bit per column, so a listed pair finds its entry by rank.  The
      // entries are read 64 at a time and kept over the chunks.
      uint32_t prev = 0xffffffffu;
      if (!first) {
        const uint32_t chunkStart = chunk * kBpChunk;
        while (qc < pe && __shfl_sync(0xffffffffu, w0, 31) < chunkStart) {
          qc += 32;
          w0 = w1;
          w1 = qc + 32 + lane < pe ? b.bpPrevCols[qc + 32 + lane] : 0xffffffffu;
        }
        const uint32_t below = __popc(__ballot_sync(0xffffffffu, w0 < chunkStart));
        const uint32_t o0 = w0 - chunkStart, o1 = w1 - chunkStart;
        const unsigned have = __reduce_or_sync(0xffffffffu, (o0 < kBpChunk ? (1u << o0) : 0u) |
                                                                (o1 < kBpChunk ? (1u << o1) : 0u));
        if ((have >> lane) & 1u) prev = qc + below + __popc(have & ((1u << lane) - 1u));
      }
      if (hit) {
        const uint32_t pos = base + count + __popc(m & ((1u << lane) - 1u));
        uint4 q;
        if (edgeRow) {
          const uint2 e = b.bpEdges[col];
          q = make_uint4(rv[0], rv[1], e.x, e.y | 0x80000000u);
        } else {
          const uint4 t = b.bpTris[col];
          q = make_uint4(rv[0], t.x, t.y, t.z);
        }
        b.contactIdx[pos] = q;
        b.contactScene[pos] = scene;
        b.bpCols[pos] = col;
        b.bpPrev[pos] = prev;
      }
      count += __popc(m);
    };
    // The count pass keeps a row's hit chunks with their masks, up to 32, so
    // that the write pass need not test the boxes again.
    uint32_t kept = 0;
    uint2 mine = make_uint2(0u, 0u);
    if constexpr (kWrite) {
      const uint32_t n = b.bpRowKept[r];
      if (n <= kBpRowHits) {
        if (lane < n) mine = b.bpRowHits[static_cast<size_t>(r) * kBpRowHits + lane];
        for (uint32_t i = 0; i < n; ++i) place(__shfl_sync(0xffffffffu, mine.x, i), __shfl_sync(0xffffffffu, mine.y, i));
        return;
      }
    }
    const float reach = bpReach(p);
    BpBox P;
    if (edgeRow) {
      P = bpLoad(b.bpEdgeBox, row.x);
    } else {
      const uint32_t vs[1] = {row.x};
      P = bpPrimitive(b, p, src, vs);
    }
    // The row's closed one-ring set: a pair whose other vertices meet it is
    // not in the superset (more than kBpClosedMax vertices: the ring lists).
    uint32_t nClosed = 0;
    {
      const uint2 r0 = b.bpRing[rv[0]];
      const uint2 r1 = edgeRow ? b.bpRing[rv[1]] : make_uint2(0u, 0u);
      nClosed = (edgeRow ? 2u : 1u) + r0.y + r1.y;
      if (nClosed <= kBpClosedMax) {
        for (uint32_t i = lane; i < nClosed; i += 32) {
          uint32_t v;
          if (i == 0) v = rv[0];
          else if (i <= r0.y) v = b.bpRingIds[r0.x + i - 1];
          else if (i == r0.y + 1) v = rv[1];
          else v = b.bpRingIds[r1.x + i - r0.y - 2];
          closedSet[warp][i] = v;
        }
      }
      __syncwarp();
    }
    auto closed = [&](uint32_t col) {
      if (nClosed > kBpClosedMax) return bpPairClosed(b, edgeRow, rv, col);
      uint32_t q0, q1, q2;
      if (edgeRow) {
        const uint2 e = b.bpEdges[col];
        q0 = e.x;
        q1 = q2 = e.y;
      } else {
        const uint4 t = b.bpTris[col];
        q0 = t.x;
        q1 = t.y;
        q2 = t.z;
      }
      for (uint32_t i = 0; i < nClosed; ++i) {
        const uint32_t v = closedSet[warp][i];
        if (v == q0 || v == q1 || v == q2) return true;
      }
      return false;
    };
    const uint32_t chunkLo = row.z / kBpChunk, chunkHi = (row.w - 1) / kBpChunk;
    const float4* superBoxes = edgeRow ? b.bpEdgeSuper : b.bpTriSuper;
    const float4* chunkBoxes = edgeRow ? b.bpEdgeChunk : b.bpTriChunk;
    const float4* primBoxes = edgeRow ? b.bpEdgeBox : b.bpTriBox;
    // Rows whose previous entries carry no lagged friction skip whole
    // superchunks whose box the row's box clears.
    bool friction = false;
    if (!first && p.ipcFriction > 0.0f)
      for (uint32_t i0 = pc; i0 < pe && !friction; i0 += 32) {
        const uint32_t i = i0 + lane;
        friction = __any_sync(0xffffffffu,
                              i < pe && b.bpPrevState[kContactStateWords * static_cast<size_t>(i) + kContactLagged].w >
                                            0.0f);
      }
    const uint32_t superLo = chunkLo / kBpChunk, superHi = chunkHi / kBpChunk;
    for (uint32_t s0 = superLo; s0 <= superHi; s0 += 32) {
      const uint32_t sc = s0 + lane;
      unsigned superTodo = __ballot_sync(0xffffffffu, sc <= superHi && (friction || !bpSeparated(
                                                                                     P, bpLoad(superBoxes, sc), reach)));
      while (superTodo) {
        const uint32_t c0 = (s0 + __ffs(superTodo) - 1) * kBpChunk;  // the superchunk's first chunk
        superTodo &= superTodo - 1;
        const uint32_t windowEnd = (c0 + 32) * kBpChunk;
        carried[warp][lane] = 0u;
        __syncwarp();
        // Previous pairs of this window that carry lagged friction and that
        // the box test leaves out stay listed.
        while (friction && pc < pe) {
          const uint32_t i = pc + lane;
          const uint32_t col = i < pe ? b.bpPrevCols[i] : 0xffffffffu;
          const bool in = i < pe && col < windowEnd;
          if (in && b.bpPrevState[kContactStateWords * static_cast<size_t>(i) + kContactLagged].w > 0.0f &&
              bpSeparated(P, bpLoad(primBoxes, col), reach))
            atomicOr(&carried[warp][col / kBpChunk - c0], 1u << (col % kBpChunk));
          const unsigned inMask = __ballot_sync(0xffffffffu, in);
          pc += __popc(inMask);
          if (inMask != 0xffffffffu) break;
        }
        __syncwarp();
        const uint32_t chunk = c0 + lane;
        const bool look = chunk >= chunkLo && chunk <= chunkHi &&
                          (carried[warp][lane] != 0u || !bpSeparated(P, bpLoad(chunkBoxes, chunk), reach));
        unsigned todo = __ballot_sync(0xffffffffu, look);
        while (todo) {
          const uint32_t j = __ffs(todo) - 1;
          todo &= todo - 1;
          const uint32_t col = (c0 + j) * kBpChunk + lane;
          bool hit = false;
          if (col >= row.z && col < row.w) {
            hit = ((carried[warp][j] >> lane) & 1u) != 0u;
            if (!hit && !bpSeparated(P, bpLoad(primBoxes, col), reach)) hit = !closed(col);
          }
          const unsigned m = __ballot_sync(0xffffffffu, hit);
          if constexpr (kWrite) {
            if (m) place(c0 + j, m);
          } else if (m) {
            if (lane == kept) mine = make_uint2(c0 + j, m);
            ++kept;
            count += __popc(m);
          }
        }
        __syncwarp();  // carried[] is rewritten by the next window
      }
    }
    if constexpr (!kWrite) {
      if (lane < kept) b.bpRowHits[static_cast<size_t>(r) * kBpRowHits + lane] = mine;
      if (lane == 0) b.bpRowKept[r] = kept;
    }
  }
  if (!kWrite && lane == 0) b.bpRowOff[r] = count;
}

constexpr int kScanThreads = 1024;

// Exclusive scan of data[0, n) in place by one block of kScanThreads threads;
// returns the total.  With the total above `limit` every entry becomes zero.
// Each warp takes a contiguous run 32 entries at a time, eight rounds in
// flight (a run per thread, entry after entry, took 60 us for 65 000 rows).
__device__ uint64_t blockScan(uint32_t* data, uint32_t n, uint64_t limit) {
  constexpr uint32_t kWarps = kScanThreads / 32, kAhead = 8;
  __shared__ uint64_t part[kWarps];
  const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x & 31u;
  const uint32_t per = ((n + kWarps - 1) / kWarps + 31u) & ~31u;
  const uint32_t lo = min(n, warp * per), hi = min(n, lo + per);
  uint64_t s = 0;
  for (uint32_t i0 = lo; i0 < hi; i0 += 32 * kAhead) {
    uint32_t v[kAhead];
#pragma unroll
    for (uint32_t j = 0; j < kAhead; ++j) v[j] = i0 + 32 * j + lane < hi ? data[i0 + 32 * j + lane] : 0u;
#pragma unroll
    for (uint32_t j = 0; j < kAhead; ++j) s += v[j];
  }
#pragma unroll
  for (uint32_t o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) part[warp] = s;
  __syncthreads();
  uint64_t run = 0, total = 0;
  for (uint32_t w = 0; w < kWarps; ++w) {
    if (w == warp) run = total;
    total += part[w];
  }
  const bool over = total > limit;
  for (uint32_t i0 = lo; i0 < hi; i0 += 32 * kAhead) {
    uint32_t v[kAhead];
#pragma unroll
    for (uint32_t j = 0; j < kAhead; ++j) v[j] = i0 + 32 * j + lane < hi ? data[i0 + 32 * j + lane] : 0u;
#pragma unroll
    for (uint32_t j = 0; j < kAhead; ++j) {
      uint32_t x = v[j];  // a run's sum may pass 32 bits only above the limit
#pragma unroll
      for (uint32_t o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      if (i0 + 32 * j + lane < hi) data[i0 + 32 * j + lane] = over ? 0u : static_cast<uint32_t>(run) + x - v[j];
      run += __shfl_sync(0xffffffffu, x, 31);
    }
  }
  __syncthreads();
  return total;
}

// Row offsets, the list's size (zero, with the overflow flags set, when it
// exceeds the capacity), each scene's span of the list, and the resets the
// static path makes in its flag and lag passes: the safe-step reductions
// every iteration, the contact alpha at the frame's first.
__global__ void __launch_bounds__(kScanThreads) bpScanKernel(Buffers b, const DevParams* __restrict__ pp,
                                                             int first) {
  const uint32_t R = b.bpRowTotal;
  const uint64_t total = blockScan(b.bpRowOff, R, b.contactCount);
  const bool over = total > b.contactCount;
  if (threadIdx.x == 0) {
    b.bpRowOff[R] = over ? 0u : static_cast<uint32_t>(total);
    b.bpStatus[0] = over ? 0u : static_cast<uint32_t>(total);
    b.bpStatus[3] = over ? 1u : 0u;
    if (over) {
      b.bpStatus[1] = 1u;
      b.bpStatus[2] = max(b.bpStatus[2], static_cast<uint32_t>(total > 0xffffffffull ? 0xffffffffull : total));
    }
  }
  __syncthreads();
  for (uint32_t s = threadIdx.x; s < b.sceneCount; s += blockDim.x) {
    const SceneRange sr = b.scenes[s];
    uint2 span = make_uint2(0u, 0u);
    if (sr.rowCount) {
      const uint32_t a = b.bpRowOff[sr.rowOff], e = b.bpRowOff[sr.rowOff + sr.rowCount];
      span = make_uint2(a, e - a);
    }
    b.bpSpan[s] = span;
    const DevParams& p = pp[s];
    if (!p.active || !p.ipc) continue;
    FrameState* fs = &b.frames[s];
    fs->stepAlphaBits = __float_as_uint(1.0f);
    fs->stepValid = 1u;
    fs->checkAlphaBits = __float_as_uint(1.0f);
    fs->checkValid = 1u;
    if (first) fs->contactAlpha = 1.0f;
  }
}

// Stable LSD radix sort of the (vertex, candidate) entries, 8 bits a pass:
// per 4096-entry tile a digit histogram, one scan of the histograms in
// digit-major order, then a scatter in which each warp ranks its entries in
// input order (match_any peers) so equal digits keep their order.
constexpr uint32_t kSortThreads = 256, kSortItems = 16, kSortTile = kSortThreads * kSortItems;

__device__ __forceinline__ uint32_t sortTiles(const uint32_t* status) {
  return (4u * __ldcg(status) + kSortTile - 1) / kSortTile;
}

__global__ void __launch_bounds__(kSortThreads) bpSortHistKernel(const uint32_t* __restrict__ keys,
                                                                 const uint32_t* status, uint32_t shift,
                                                                 uint32_t* __restrict__ hist) {
  __shared__ uint32_t h[256];
  const uint32_t M = 4u * __ldcg(status), tiles = sortTiles(status);
  if (blockIdx.x >= tiles) return;
  h[threadIdx.x] = 0u;
  __syncthreads();
#pragma unroll
  for (uint32_t j = 0; j < kSortItems; ++j) {
    const uint32_t i = blockIdx.x * kSortTile + j * kSortThreads + threadIdx.x;
    if (i < M) atomicAdd(&h[(keys[i] >> shift) & 255u], 1u);
  }
  __syncthreads();
  hist[threadIdx.x * tiles + blockIdx.x] = h[threadIdx.x];
}

// One block per digit: the exclusive scan of the digit's tile counts and the
// digit's total (after the 256 x tiles histogram).
__global__ void __launch_bounds__(kScanThreads) bpSortScanKernel(const uint32_t* status, uint32_t* hist) {
  const uint32_t tiles = sortTiles(status);
  const uint64_t total = blockScan(hist + static_cast<size_t>(blockIdx.x) * tiles, tiles, ~0ull);
  if (threadIdx.x == 0) hist[256u * tiles + blockIdx.x] = static_cast<uint32_t>(total);
}

// kFirst: the entries still lie four to a candidate, in candidate order, so
// their values are not stored.
template <bool kFirst>
__global__ void __launch_bounds__(kSortThreads) bpSortScatterKernel(const uint32_t* __restrict__ kin,
                                                                    const uint32_t* __restrict__ vin,
                                                                    uint32_t* __restrict__ kout,
                                                                    uint32_t* __restrict__ vout,
                                                                    const uint32_t* status, uint32_t shift,
                                                                    const uint32_t* __restrict__ hist) {
  __shared__ uint32_t wh[kSortThreads / 32][256];
  __shared__ uint32_t digitBase[256];
  const uint32_t M = 4u * __ldcg(status), tiles = sortTiles(status);
  const uint32_t tile = blockIdx.x;
  if (tile >= tiles) return;
  const uint32_t w = threadIdx.x / 32, lane = threadIdx.x & 31u;
  for (uint32_t d = threadIdx.x; d < 256u * (kSortThreads / 32); d += kSortThreads) (&wh[0][0])[d] = 0u;
  // Exclusive prefix of the digit totals (one digit per thread).
  digitBase[threadIdx.x] = hist[256u * tiles + threadIdx.x];
  __syncthreads();
  for (uint32_t o = 1; o < 256u; o <<= 1) {
    const uint32_t add = threadIdx.x >= o ? digitBase[threadIdx.x - o] : 0u;
    __syncthreads();
    digitBase[threadIdx.x] += add;
    __syncthreads();
  }
  const uint32_t mine = digitBase[threadIdx.x] - hist[256u * tiles + threadIdx.x];
  __syncthreads();
  digitBase[threadIdx.x] = mine;
  __syncthreads();
  const uint32_t base = tile * kSortTile + w * (kSortItems * 32);
  uint32_t dig[kSortItems], pos[kSortItems];
#pragma unroll
  for (uint32_t j = 0; j < kSortItems; ++j) {
    const uint32_t i = base + j * 32 + lane;
    const bool valid = i < M;
    const uint32_t d = valid ? (kin[i] >> shift) & 255u : 256u;
    const unsigned peers = __match_any_sync(0xffffffffu, d);
    const uint32_t rank = __popc(peers & ((1u << lane) - 1u));
    const uint32_t before = valid ? wh[w][d] : 0u;
    __syncwarp();
    if (valid && rank == 0) wh[w][d] = before + __popc(peers);
    __syncwarp();
    dig[j] = d;
    pos[j] = before + rank;
  }
  __syncthreads();
  {
    const uint32_t d = threadIdx.x;  // one digit per thread
    uint32_t run = 0;
#pragma unroll
    for (uint32_t ww = 0; ww < kSortThreads / 32; ++ww) {
      const uint32_t t = wh[ww][d];
      wh[ww][d] = run;
      run += t;
    }
  }
  __syncthreads();
#pragma unroll
  for (uint32_t j = 0; j < kSortItems; ++j) {
    if (dig[j] < 256u) {
      const uint32_t i = base + j * 32 + lane;
      const uint32_t o = digitBase[dig[j]] + hist[dig[j] * tiles + tile] + wh[w][dig[j]] + pos[j];
      kout[o] = kin[i];
      vout[o] = kFirst ? i / 4u : vin[i];
    }
  }
}

// Each vertex's run of the sorted keys is its active row: the run's first
// entry sets its start, and first and last add up its length (integers, on the
// zero the boxes pass left).
__global__ void __launch_bounds__(kBlock) bpSegmentsKernel(Buffers b, const uint32_t* __restrict__ keys) {
  const uint32_t n = __ldcg(b.bpStatus);  // groups of four entries
  for (uint32_t g = blockIdx.x * kBlock + threadIdx.x; g < n; g += gridDim.x * kBlock) {
    const uint4 q = reinterpret_cast<const uint4*>(keys)[g];
    const uint32_t before = g > 0 ? keys[4 * g - 1] : ~0u, after = g + 1 < n ? keys[4 * g + 4] : ~0u;
    const uint32_t k[6] = {before, q.x, q.y, q.z, q.w, after};
#pragma unroll
    for (uint32_t j = 1; j <= 4; ++j) {
      if (k[j] >= b.bpSentinel) continue;
      const uint32_t i = 4 * g + j - 1;
      if (k[j - 1] != k[j]) {
        b.contactRange[k[j]] = make_uint2(i, 0u);
        atomicSub(&b.activeCount[k[j]], i);
      }
      if (k[j + 1] != k[j]) atomicAdd(&b.activeCount[k[j]], i + 1);
    }
  }
}

// ---------------------------------------------------------------------------
// The per-vertex JGS2 local solve, stable Neo-Hookean path
// (jgs2Solve, jgs2-shader.ts:2991-3473).  W lanes cooperate on one vertex:
// item u < K is cubature record u, item u >= K is incident tet u - K; lane j
// takes items j, j + W, ...  Cubature record state is cached in shared memory
// for the line search; incident deformation gradients are recomputed per
// trial from L1-resident data.
struct CubState {
  M3 F;
  float I0, J0;
  M3 dF0, dF1, dF2;
  float3 gQ;
  S3 HQ;
  float w, vol, lambda, mu;
  uint32_t slot;
  float3 gs;
};
static_assert(sizeof(CubState) <= kRecFloats * 4, "cubature cache record too small");

#ifndef JGS2_SOLVE_STAGE
#define JGS2_SOLVE_STAGE 1
#endif
// Shared-memory slot of one cubature record of a solve block.  The block
// first stages every record's header, basis blocks and tetrahedron record
// into its slot with asynchronous copies (all independent, so the whole
// block's input is in flight at once instead of one dependent chain per
// record and lane); the lane that owns the record then reads its inputs from
// the slot and overwrites the slot with the record's cached state for the
// line search.
struct RecSlot {
  uint4 head[2];   // (tet, weight bits, 0, 0), the tet's vertex indices
  float4 basis[9]; // 36 floats: four row-major 3x3 blocks
  float4 tet[4];   // [g1 vol] [g2 lambda] [g3 mu] [indices]
};
static_assert(sizeof(CubState) <= sizeof(RecSlot), "record state must fit its staging slot");
// Records per vertex up to this many bytes of cached state are cached in
// shared memory (K <= 68 with staging); wider ones are recomputed per trial.
#ifndef JGS2_SOLVE_CACHE_BYTES
#define JGS2_SOLVE_CACHE_BYTES 16384
#endif
constexpr size_t kSolveCacheBytesPerVertex = JGS2_SOLVE_CACHE_BYTES;
#if JGS2_SOLVE_STAGE
constexpr size_t kSolveSlotBytes = sizeof(RecSlot);
#else
constexpr size_t kSolveSlotBytes = sizeof(CubState);
#endif

__device__ __forceinline__ void cpAsync16(void* smem, const void* gmem) {
  const uint32_t sa = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cpAsyncWaitAll() {
  asm volatile("cp.async.commit_group;" ::: "memory");
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}
__device__ __forceinline__ TetRec tetFromSlot(const float4* q) {
  const float4 a = q[0], b = q[1], c = q[2];
  const float4 d = q[3];
  TetRec r;
  r.g1 = f3(a.x, a.y, a.z);
  r.g2 = f3(b.x, b.y, b.z);
  r.g3 = f3(c.x, c.y, c.z);
  r.vol = a.w;
  r.lambda = b.w;
  r.mu = c.w;
  r.idx = make_uint4(__float_as_uint(d.x), __float_as_uint(d.y), __float_as_uint(d.z), __float_as_uint(d.w));
  return r;
}
// loadBlockVec from a shared-memory copy of the record's basis.
__device__ __forceinline__ M3 loadBlockVecShared(const float4* rec, int l) {
  const int k0 = (9 * l) >> 2;
  const int off = 9 * l - 4 * k0;
  const float4 a = rec[k0], b = rec[k0 + 1], c = rec[k0 + 2];
  const float f[12] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x, c.y, c.z, c.w};
  return {f3(f[off + 0], f[off + 3], f[off + 6]), f3(f[off + 1], f[off + 4], f[off + 7]),
          f3(f[off + 2], f[off + 5], f[off + 8])};
}

#ifndef JGS2_SOLVE_MIN_BLOCKS
#define JGS2_SOLVE_MIN_BLOCKS 4
#endif

// kExt: some scene of the engine has cloth or contact candidates (their
// gathers and line search terms are compiled out otherwise).
// State of cubature record `rec` of vertex v (jgs2-shader.ts:3197-3263), all
// in the source vertex's frame: the record tet's deformation gradient F and
// its invariants, the projected directions dF_c = sum_l B'_l[:,c] g_l^T with
// B'_l = R_l Ubar_l, the inertia / objective quadratic (gQ, HQ), the weight,
// the tet's material and, when v is one of the tet's vertices, its slot and
// shape gradient.  Read from the block's staged slot or from global memory;
// st.w = 0 for an empty record.  `r` receives the record's tet.
template <bool kCoherent, class Basis>
__device__ __forceinline__ void recordStateOf(const Buffers& b, const DevParams& p, uint32_t v, float w, const uint4& idx,
                                              const TetRec& r, Basis basis, const float4* __restrict__ src,
                                              bool objActive, CubState& st) {
  M3 F = mzero(), dF0 = mzero(), dF1 = mzero(), dF2 = mzero();
  float3 gQ = f3(0, 0, 0);
  S3 HQ = szero();
  uint32_t slot = 4;
  float3 x0 = f3(0, 0, 0);
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    const uint32_t q = idxAt(idx, l);
    if (q == v) slot = l;
    const float3 gl = shapeGradient(r, l);
    VertexPack pk;
    if constexpr (kCoherent) {
      const float4 pq = b.predicted[q];
      pk = {loadFrameT<true>(b.vertexPack, q), xyz(__ldca(src + q)), xyz(pq), pq.w};
    } else {
      pk = loadPack(b.vertexPack, q);
    }
    const M3 B = mm(pk.R, basis(l));
    const float3 xl = pk.x;
    if (l == 0) x0 = xl;
    if (l > 0) F = F + outer(xl - x0, gl);
    dF0 = dF0 + outer(B.c0, gl);
    dF1 = dF1 + outer(B.c1, gl);
    dF2 = dF2 + outer(B.c2, gl);
    // The distributed inertia weight is 0 when pinned.
    const float dW = pk.dW;
    float3 lin = dW * (xl - pk.pred);
    float quad = dW;
    const uint4 qi = objActive ? b.vinfo[q] : make_uint4(0u, 0u, 1u, 0u);
    if (objActive && !isPinned(qi)) {
      const float nq = float(qi.y > 1u ? qi.y : 1u);
      lin = lin + objectiveGradient(p, b, q, xl) * (1.0f / nq);
      quad += targetStiffness(p, b, q) / nq;
    }
    gQ = gQ + mtv(B, lin);
    saddScaled(HQ, quad, gramColumns(B));
  }
  st.F = F;
  st.I0 = frob(F, F);
  st.J0 = mdet(F);
  st.dF0 = dF0; st.dF1 = dF1; st.dF2 = dF2;
  st.gQ = gQ;
  st.HQ = HQ;
  st.w = w;
  st.vol = r.vol; st.lambda = r.lambda; st.mu = r.mu;
  st.slot = slot;
  st.gs = slot < 4 ? shapeGradient(r, slot) : f3(0, 0, 0);
}

template <bool kCoherent, bool kStaged>
__device__ __forceinline__ void recordState(const Buffers& b, const DevParams& p, uint32_t v, size_t rec,
                                            const RecSlot* staged, const float4* __restrict__ src, bool objActive,
                                            CubState& st, TetRec& r) {
  uint4 head, idx;
  if constexpr (kStaged) {
    head = staged->head[0];
    idx = staged->head[1];
  } else {
    head = __ldg(&b.cubHead[2 * rec]);
    idx = __ldg(&b.cubHead[2 * rec + 1]);
  }
  const uint32_t t = head.x;
  const float w = __uint_as_float(head.y);
  st.w = 0.0f;
  // Headers hold global tet ids; out-of-range records were emptied at create.
  if (!(t != kEmptyTet && w > 0.0f)) return;
  if (!inBounds(t, b.tetTotal, kSiteRecordTet) || !inBounds(idx.x, b.vertexTotal, kSiteRecordVertex) ||
      !inBounds(idx.y, b.vertexTotal, kSiteRecordVertex) || !inBounds(idx.z, b.vertexTotal, kSiteRecordVertex) ||
      !inBounds(idx.w, b.vertexTotal, kSiteRecordVertex))
    return;
  if constexpr (kStaged) {
    r = tetFromSlot(staged->tet);
    recordStateOf<kCoherent>(b, p, v, w, idx, r, [&](int l) { return loadBlockVecShared(staged->basis, l); }, src,
                             objActive, st);
  } else {
    r = loadTet(b.tets, t);
    const float4* U = b.cubBasis + 9ull * rec;
    recordStateOf<kCoherent>(b, p, v, w, idx, r, [&](int l) { return loadBlockVec(U, l); }, src, objActive, st);
  }
}

// One block's chunk `chunk` of the vertex list: vertices
// [chunk * groupsPerBlock, (chunk + 1) * groupsPerBlock) of `list` (or of all
// vertices).  Every thread of the block calls it with the same chunk.
template <int W, bool kExt, bool kCoherent = false, bool kCache = true>
__device__ __forceinline__ void solveChunk(const Buffers& b, const DevParams* __restrict__ pp,
                                           const float4* __restrict__ src, float4* tgt,
                                           const uint32_t* __restrict__ list, uint32_t count, uint32_t K,
                                           int cachedIncident, uint32_t groupsPerBlock, uint32_t chunk) {
  extern __shared__ float4 cache4[];
  unsigned char* slotBase = reinterpret_cast<unsigned char*>(cache4);
  __shared__ uint32_t sFail, sMaxBack, sSkip, sEvals, sMaxShift, sValid, sScene;
  // Lane groups never straddle a warp: warp w holds groups w * (32 / W) ...;
  // lanes past the warp's last whole group, or past groupsPerBlock, are idle.
  constexpr uint32_t kGroupsPerWarp = 32 / W;
  const uint32_t lane = (threadIdx.x & 31u) % W;
  const uint32_t groupInWarp = (threadIdx.x & 31u) / W;
  const uint32_t group = (threadIdx.x >> 5) * kGroupsPerWarp + groupInWarp;
  const bool groupLane = groupInWarp < kGroupsPerWarp && group < groupsPerBlock;
  const unsigned mask = W == 32 ? 0xffffffffu : (((1u << W) - 1u) << (groupInWarp * W));
  if (threadIdx.x == 0) {
    sFail = 0; sMaxBack = 0; sSkip = 0; sEvals = 0; sMaxShift = 0; sValid = 1;
    const uint32_t first = chunk * groupsPerBlock;
    sScene = b.vertexScene[list ? list[first] : first];
  }
  __syncthreads();
#if JGS2_SOLVE_STAGE
  if constexpr (kCache) {
    // Stage the block's records: headers and basis blocks, then (once the
    // headers have landed) the tetrahedron records they name.
    RecSlot* slots = reinterpret_cast<RecSlot*>(slotBase);
    const uint32_t nrec = groupsPerBlock * K;
    // Sixteen-byte chunks in address order: a record's two header chunks and
    // nine basis chunks are consecutive, so a warp's copies are coalesced.
    for (uint32_t c = threadIdx.x; c < nrec * 11u; c += blockDim.x) {
      const uint32_t r = c / 11u, part = c - r * 11u;
      const uint32_t g = r / K, it = chunk * groupsPerBlock + g;
      if (it >= count) continue;
      const uint32_t sv = list ? list[it] : it;
      if (!inBounds(sv, b.vertexTotal, kSiteListVertex)) continue;
      const size_t rec = static_cast<size_t>(sv) * K + (r - g * K);
      if (part < 2u) cpAsync16(&slots[r].head[part], &b.cubHead[2 * rec + part]);
      else cpAsync16(&slots[r].basis[part - 2u], &b.cubBasis[9 * rec + (part - 2u)]);
    }
    cpAsyncWaitAll();
    __syncthreads();
    for (uint32_t c = threadIdx.x; c < nrec * 4u; c += blockDim.x) {
      const uint32_t r = c >> 2, part = c & 3u;
      if (chunk * groupsPerBlock + r / K >= count) continue;
      const uint4 head = slots[r].head[0];
      if (head.x != kEmptyTet && __uint_as_float(head.y) > 0.0f && inBounds(head.x, b.tetTotal, kSiteRecordTet))
        cpAsync16(&slots[r].tet[part], &b.tets[4ull * head.x + part]);
    }
    cpAsyncWaitAll();
    __syncthreads();
  }
#endif
  // One vertex per lane group; its scene selects the settings and records.
  const uint32_t item = chunk * groupsPerBlock + group;
  const uint32_t listed = (groupLane && item < count) ? (list ? list[item] : item) : 0u;
  const bool haveVertex = groupLane && item < count && inBounds(listed, b.vertexTotal, kSiteListVertex);
  const uint32_t v = haveVertex ? listed : 0u;
  const uint32_t scene = haveVertex ? b.vertexScene[v] : sScene;
  // Per-vertex outputs owned by lane 0.
  uint32_t status = kNonfinite, backtracks = 0, evals = 0;
  float shiftN = 0.0f;
  bool localValid = true, haveRecord = false;
  if (haveVertex && pp[scene].active) {
    const DevParams p = pp[scene];
    FrameState* fs = &b.frames[scene];
    const bool isLatched = latched(p, fs);
    const uint4 info = b.vinfo[v];
    const float4 rm = b.restMass[v];
    if (isLatched) {
      if (lane == 0) tgt[v] = ldPos<kCoherent>(src, v);
    } else if (isPinned(info)) {
      if (lane == 0) {
        tgt[v] = make_float4(rm.x, rm.y, rm.z, 1.0f);
        b.finalUpdate[v] = 0.0f;
        float4* L = &b.local[4ull * v];
        L[0] = L[1] = L[2] = make_float4(0, 0, 0, 0);
        L[3] = make_float4(0, 0, 0, float(kPinned));
        status = kPinned;
        haveRecord = true;
      }
    } else {
      const float4 c0 = fs->control[0];
      const uint32_t vb = controlBits(c0.w) & kValidityMask;
      const bool amv = (vb & kAcceptedMinimumValid) != 0u && finiteS(c0.z);
      if (!(amv && c0.z > kDeterminantFloor)) {
        // Preflight rejection before any material evaluation (jgs2-shader.ts:3042-3081).
        if (lane == 0) {
          tgt[v] = ldPos<kCoherent>(src, v);
          b.finalUpdate[v] = 0.0f;
          float4* L = &b.local[4ull * v];
          L[0] = L[1] = L[2] = make_float4(0, 0, 0, 0);
          status = amv ? kLineSearchFailed : kNonfinite;
          L[3] = make_float4(amv ? c0.z : 0.f, 0, 0, float(status));
          localValid = status != kNonfinite;
          haveRecord = true;
        }
      } else {
        const float3 position = xyz(ldPos<kCoherent>(src, v));
        const float3 predV = xyz(b.predicted[v]);
        const float inertia = rm.w * p.invDt2;
        const float dWs = distributedInertiaWeight(rm, info, p.invDt2);
        const float nS = float(info.y > 1u ? info.y : 1u);
        const bool objActive = p.objectiveFlags != 0u;
        const float3 objS = objActive ? objectiveGradient(p, b, v, position) : f3(0, 0, 0);
        const float ktS = targetStiffness(p, b, v);
        Comp3 gsum = czero();  // compensated gradient gather
        S3 hess = szero();
        // Record terms are formed in the source vertex's frame: with
        // B_l = R_l Ubar_l R_s^T = B'_l R_s^T, a record's projected gradient
        // and Hessian are R_s g' and R_s H' R_s^T of the same expressions over
        // B'_l = R_l Ubar_l, so R_s is applied once per record instead of once
        // per basis block.  The exact source block subtracted for a record at
        // the vertex's own slot is formed in the world frame.
        const M3 Rs = loadFrameT<kCoherent>(b.vertexPack, v);
        unsigned char* mySlots = slotBase + static_cast<size_t>(group) * K * kSolveSlotBytes;
        // Cubature records first, then (unless cached) the incident tets, in
        // separate loops so the two kinds of item never share a divergent pass.
        for (uint32_t u = lane; u < K; u += W) {
          // ---- cubature record (jgs2-shader.ts:3197-3263) ----
          CubState st;
          TetRec r;
          const size_t rec = static_cast<size_t>(v) * K + u;
          if constexpr (kCache && JGS2_SOLVE_STAGE)
            recordState<kCoherent, true>(b, p, v, rec, reinterpret_cast<const RecSlot*>(mySlots + u * kSolveSlotBytes),
                                         src, objActive, st, r);
          else
            recordState<kCoherent, false>(b, p, v, rec, nullptr, src, objActive, st, r);
          if (st.w > 0.0f) {
            const float w = st.w;
            const M3& F = st.F;
            const M3 &dF0 = st.dF0, &dF1 = st.dF1, &dF2 = st.dF2;
            const PiolaTerms pt = piolaTerms(F, r.lambda, r.mu);
            const M3 P = piola(F, pt);
            float3 pg = r.vol * f3(frob(dF0, P), frob(dF1, P), frob(dF2, P)) + st.gQ;
            // Reduced material Hessian vol <dF_r, DP[dF_c]>; the cofactor
            // term <A, Dcof[B]> is symmetric, so one directional cofactor is
            // live at a time.
            const float p0 = frob(F, dF0), p1 = frob(F, dF1), p2 = frob(F, dF2);
            const float q0 = frob(pt.cof, dF0), q1 = frob(pt.cof, dF1), q2 = frob(pt.cof, dF2);
            S3 ph;
            {
              const M3 D0 = dcofactor(F, dF0);
              ph.xx = pt.b * frob(dF0, D0);
              ph.xy = pt.b * frob(dF1, D0);
              ph.xz = pt.b * frob(dF2, D0);
            }
            {
              const M3 D1 = dcofactor(F, dF1);
              ph.yy = pt.b * frob(dF1, D1);
              ph.yz = pt.b * frob(dF2, D1);
            }
            ph.zz = pt.b * frob(dF2, dcofactor(F, dF2));
            ph.xx += pt.a * frob(dF0, dF0) + pt.c1 * p0 * p0 + r.lambda * q0 * q0;
            ph.yy += pt.a * frob(dF1, dF1) + pt.c1 * p1 * p1 + r.lambda * q1 * q1;
            ph.zz += pt.a * frob(dF2, dF2) + pt.c1 * p2 * p2 + r.lambda * q2 * q2;
            ph.xy += pt.a * frob(dF0, dF1) + pt.c1 * p0 * p1 + r.lambda * q0 * q1;
            ph.xz += pt.a * frob(dF0, dF2) + pt.c1 * p0 * p2 + r.lambda * q0 * q2;
            ph.yz += pt.a * frob(dF1, dF2) + pt.c1 * p1 * p2 + r.lambda * q1 * q2;
            ph.xx *= r.vol; ph.yy *= r.vol; ph.zz *= r.vol; ph.xy *= r.vol; ph.xz *= r.vol; ph.yz *= r.vol;
            sadd(ph, st.HQ);
            cadd(gsum, w * mv(Rs, pg));
            saddScaled(hess, w, srotate(Rs, ph));
            if (st.slot < 4) {
              // Remove the exact source block already in the local gather.
              const float3 gs = st.gs;
              float3 ps = r.vol * mv(P, gs) + dWs * (position - predV);
              if (objActive) ps = ps + objS * (1.0f / nS);
              const float3 u1 = mv(F, gs), w1 = mv(pt.cof, gs);
              S3 blk = szero();
              saddDiag(blk, pt.a * dot3(gs, gs));
              saddOuter(blk, pt.c1, u1);
              saddOuter(blk, r.lambda, w1);
              cadd(gsum, (-w) * ps);
              saddScaled(hess, -w * r.vol, blk);
              saddDiag(hess, -w * (dWs + ktS / nS));
            }
          }
          if constexpr (kCache) *reinterpret_cast<CubState*>(mySlots + u * kSolveSlotBytes) = st;
        }
        if (!cachedIncident) {
          for (uint32_t a = lane; a < info.y; a += W) {
            // ---- incident tetrahedron (jgs2-shader.ts:3097-3111) ----
            const uint32_t entry = __ldg(&b.adjacency[info.x + a]);
            TetRec r;
            if (!incidentTetChecked(b.tets, entry, b.tetTotal, b.vertexTotal, &r)) continue;
            const M3 F = deformationAtT<kCoherent>(r, src);
            const PiolaTerms pt = piolaTerms(F, r.lambda, r.mu);
            const float3 g = shapeGradient(r, entry & 3u);
            cadd(gsum, r.vol * mv(piola(F, pt), g));
            addIncidentBlock(hess, r, F, pt, g);
          }
          // ---- cloth membrane and bending (jgs2-shader.ts:3113-3186) ----
          if (kExt && p.cloth)
            clothLocalSystem<true, kCoherent>(b.clothTris, b.clothHinges, b.clothIncidence, b.clothRange[v], src,
                                   clothMaterial(p), lane, W, gsum, hess);
        }
        // ---- IPC contact (jgs2-shader.ts:3193-3195): the cached source
        // contacts, or fresh ones under the coloured schedule ----
        if (kExt && p.ipc)
          contactLocal<true>(b, p, v, src, !cachedIncident, kContactSource, b.contactNear, lane, W, gsum, hess);
        // Group reduction of the gather.
        groupMerge<W>(gsum, mask);
        hess.xx = groupSum<W>(hess.xx, mask);
        hess.yy = groupSum<W>(hess.yy, mask);
        hess.zz = groupSum<W>(hess.zz, mask);
        hess.xy = groupSum<W>(hess.xy, mask);
        hess.xz = groupSum<W>(hess.xz, mask);
        hess.yz = groupSum<W>(hess.yz, mask);
        if (cachedIncident) {
          const float4 i0 = b.incident[3ull * v], i1 = b.incident[3ull * v + 1], i2 = b.incident[3ull * v + 2];
          cadd(gsum, f3(i0.x, i0.y, i0.z));
          hess.xx += i0.w;
          hess.yy += i1.x;
          hess.zz += i1.y;
          hess.xy += i1.z;
          hess.xz += i1.w;
          hess.yz += i2.x;
        }
        // Own terms: inertia, objectives, floor (jgs2-shader.ts:3083-3092, 3188-3191).
        cadd(gsum, inertia * (position - predV));
        saddDiag(hess, inertia);
        if (objActive) cadd(gsum, objS);
        if (p.objectiveFlags & 2u) saddDiag(hess, ktS);
        if (p.floorStiffness > 0.0f && position.y < p.floorHeight) {
          cadd(gsum, f3(0.0f, p.floorStiffness * (position.y - p.floorHeight), 0.0f));
          hess.yy += p.floorStiffness;
        }
        const float3 grad = cvalue(gsum);
        // ---- globalization and line search (jgs2-shader.ts:3265-3473) ----
        const SolveResult dr = globalizationSolve(hess, grad, inertia);
        status = kNonfinite;
        const float3 fullP = position + dr.direction;
        const float3 fullD = fullP - position;
        const float scs = fmaxf(fabsf(position.x), fmaxf(fabsf(position.y), fabsf(position.z)));
        const float resolution =
            fmaxf(p.sceneScale, fmaxf(scs, 1.0e-12f)) * kUnitRoundoff * kPositionResolutionMultiplier;
        const bool below = dr.status == kAccepted && finiteV(fullP) && finiteV(fullD) && scaledLength(fullD) <= resolution;
        if (dr.status == kAccepted) status = below ? kZeroGradient : kLineSearchFailed;
        else if (dr.status == kZeroGradient) status = kZeroGradient;
        else if (dr.status == kShiftLimit) status = kShiftLimit;
        else if (dr.status == kCholeskyFailed) status = kCholeskyFailed;
        else if (dr.status == kNonDescent) status = kNonDescent;
        float alpha = 0.0f, acceptedDelta = 0.0f, bound = 0.0f, minTrialDet = 0.0f;
        float3 acceptedD = f3(0, 0, 0), acceptedP = position;
        if (dr.status == kAccepted && !below) {
          float ta = 1.0f;
          const float dl = scaledLength(dr.direction);
          if (p.maxStep > 0.0f && dl > p.maxStep) ta = p.maxStep / dl;
          const float controlMin = c0.z;  // accepted-source minimum (finite here)
          const uint4 cr = (kExt && p.cloth) ? b.clothRange[v] : make_uint4(0u, 0u, 0u, 0u);
          const uint32_t contactFirst = (kExt && p.ipc) ? b.contactRange[v].x : 0u;
          const uint32_t contactActive = (kExt && p.ipc) ? b.activeCount[v] : 0u;
          const ClothMaterial cmat = clothMaterial(p);
          for (uint32_t bt = 0; bt <= kMaxBacktracks; ++bt) {
            const float3 tp = position + ta * dr.direction;
            const float3 td = tp - position;
            if (!finiteV(tp) || !finiteV(td)) { status = kNonfinite; minTrialDet = 0.f; backtracks = bt; break; }
            const float tl = scaledLength(td);
            if (p.maxStep > 0.0f && tl > p.maxStep) { ta *= kBacktrackFactor; continue; }
            if (tl <= resolution) { status = kZeroGradient; minTrialDet = 0.f; backtracks = bt; break; }
            const float gd = dot3(grad, td);
            if (!finiteS(gd)) { status = kNonfinite; minTrialDet = 0.f; backtracks = bt; break; }
            if (!(gd < 0.0f)) { status = kZeroGradient; minTrialDet = 0.f; backtracks = bt; break; }
            // Restricted geometry and energy in one pass over the items
            // (restrictedMinimumDeformationDeterminant :1980-2118 and
            // restrictedEnergyDelta :2120-2337); the energy is used only
            // when the geometry is feasible, as in the reference order.
            float jmin = kF32Max, de = 0.0f;
            const float3 ts = mtv(Rs, td);
            bool geomFinite = true;
            // A lane's items in order: its cached cubature records, then its
            // incident tets (the same per-lane order as one merged loop).
            for (uint32_t u = lane; u < K; u += W) {
              CubState stLocal;
              if constexpr (!kCache) {
                // No shared cache for wide records: recompute the record's
                // state (the same arithmetic as the gather above).
                TetRec rr;
                recordState<kCoherent, false>(b, p, v, static_cast<size_t>(v) * K + u, nullptr, src, objActive,
                                              stLocal, rr);
              }
              const CubState& st =
                  kCache ? *reinterpret_cast<const CubState*>(mySlots + u * kSolveSlotBytes) : stLocal;
              if (!(st.w > 0.0f)) continue;
              float J = 0.0f;
              // Record state is in the source frame: the trial step there is R_s^T td.
              const M3 D = ts.x * st.dF0 + ts.y * st.dF1 + ts.z * st.dF2;
              const float dm = st.vol * snhEnergyDelta(st.F, st.I0, st.J0, D, st.lambda, st.mu, &J);
              float comp = dm + dot3(ts, st.gQ) + 0.5f * dot3(ts, smv(st.HQ, ts));
              if (st.slot < 4) {
                float Js;
                comp -= st.vol * snhEnergyDelta(st.F, st.I0, st.J0, outer(td, st.gs), st.lambda, st.mu, &Js);
                comp -= dWs * (dot3(position - predV, td) + 0.5f * dot3(td, td));
                if (objActive) comp -= objectiveDelta(p, b, v, position, td) / nS;
              }
              de += st.w * comp;
              if (!finiteS(J)) geomFinite = false;
              jmin = fminf(jmin, J);
            }
            // Incident tets of lane-order index u >= K, i.e. adjacency slot u - K.
            const uint32_t firstInc = lane >= K % W ? lane - K % W : lane + W - K % W;
#if JGS2_CONV_LOOKAHEAD
            // The lane's next incident tet is requested before the current
            // one's arithmetic (as in the convergence gather).
            uint32_t nextEntry = firstInc < info.y ? __ldg(&b.adjacency[info.x + firstInc]) : 0u;
            TetRec nextRec;
            bool nextOk = false;
            if (firstInc < info.y) nextOk = incidentTetChecked(b.tets, nextEntry, b.tetTotal, b.vertexTotal, &nextRec);
#endif
            for (uint32_t a = firstInc; a < info.y; a += W) {
              float J = 0.0f;
#if JGS2_CONV_LOOKAHEAD
              const uint32_t entry = nextEntry;
              const TetRec r = nextRec;
              const bool tetOk = nextOk;
              if (a + W < info.y) {
                nextEntry = __ldg(&b.adjacency[info.x + a + W]);
                nextOk = incidentTetChecked(b.tets, nextEntry, b.tetTotal, b.vertexTotal, &nextRec);
              }
#else
              const uint32_t entry = __ldg(&b.adjacency[info.x + a]);
              TetRec r;
              const bool tetOk = incidentTetChecked(b.tets, entry, b.tetTotal, b.vertexTotal, &r);
#endif
              if (!tetOk) continue;
              const M3 F = deformationAtT<kCoherent>(r, src);
              const float I0 = frob(F, F);
              const float J0 = mdet(F);
#if JGS2_LS_RANK1
              de += r.vol * snhEnergyDeltaRankOne(F, I0, J0, td, shapeGradient(r, entry & 3u), r.lambda, r.mu, &J);
#else
              de += r.vol * snhEnergyDelta(F, I0, J0, outer(td, shapeGradient(r, entry & 3u)), r.lambda, r.mu, &J);
#endif
              if (!finiteS(J)) geomFinite = false;
              jmin = fminf(jmin, J);
            }
            // Cloth: signed area stretch at the source and the trial pose
            // (jgs2-shader.ts:2067-2116) and the membrane / bending energy
            // deltas (:2207-2263) of the incident elements.
            const float3 trialPos = position + td;
            for (uint32_t a = lane; a < cr.y; a += W) {
              const uint32_t entry = __ldg(&b.clothIncidence[cr.x + a]);
              const uint32_t slot = entry & 3u;
              const ClothTri ct = loadClothTri(b.clothTris, entry >> 2);
              const float3 x0 = xyz(ldPos<kCoherent>(src, ct.i0)), x1 = xyz(ldPos<kCoherent>(src, ct.i1)), x2 = xyz(ldPos<kCoherent>(src, ct.i2));
              const float3 y0 = slot == 0u ? trialPos : x0;
              const float3 y1 = slot == 1u ? trialPos : x1;
              const float3 y2 = slot == 2u ? trialPos : x2;
              const float3 sn = clothRawNormal(x0, x1, x2), tn = clothRawNormal(y0, y1, y2);
              const float twice = 2.0f * ct.area;
              const float ss = length3(sn) / twice, tm = length3(tn) / twice;
              const float ts = dot3(sn, tn) > 0.0f ? tm : -tm;
              if (!(twice > 0.0f) || !finiteS(ss) || !finiteS(ts)) geomFinite = false;
              jmin = fminf(jmin, fminf(ss, ts));
              de += clothMembraneEnergy(ct, y0, y1, y2, cmat) - clothMembraneEnergy(ct, x0, x1, x2, cmat);
            }
            for (uint32_t a = lane; a < cr.w; a += W) {
              const uint32_t entry = __ldg(&b.clothIncidence[cr.z + a]);
              const uint32_t slot = entry & 3u, h = entry >> 2;
              const uint4 q = hingeIndices(b.clothHinges, h);
              const float4 rest = __ldg(&b.clothHinges[2ull * h + 1]);
              const float3 x0 = xyz(ldPos<kCoherent>(src, q.x)), x1 = xyz(ldPos<kCoherent>(src, q.y)), x2 = xyz(ldPos<kCoherent>(src, q.z)), x3 = xyz(ldPos<kCoherent>(src, q.w));
              const float es = clothBendingEnergy(x0, x1, x2, x3, rest, cmat.bending);
              const float et = clothBendingEnergy(slot == 0u ? trialPos : x0, slot == 1u ? trialPos : x1,
                                                  slot == 2u ? trialPos : x2, slot == 3u ? trialPos : x3, rest,
                                                  cmat.bending);
              de += et - es;
            }
            // IPC: a trial within the minimum distance of an active candidate
            // is infeasible (jgs2-shader.ts:1997-2038); barrier and lagged
            // friction energy deltas (:2137-2196).
            if (kExt && contactActive) {
              const float dl = length3(td);
              ContactBatch batch;
              for (uint32_t a = lane; a < contactActive; a += W) {
                uint32_t c;
                if (!cachedIncident) {
                  c = b.activeIds[contactFirst + a];
                } else {
                  const float near = batch.next(b.activeIds + contactFirst, b.contactNear, a, contactActive, W, &c);
                  if (!ipcNearValid(near)) {
                    geomFinite = false;
                    continue;
                  }
                  const float left = fabsf(near) - dl;
                  if (left > p.ipcMinDistance && !(left < p.ipcActivation) && !ipcNearFriction(near)) continue;
                }
                const float4* cst = b.contactState + kContactStateWords * static_cast<size_t>(c);
                const ContactData source = cachedIncident ? ipcCached(cst[kContactSource], cst[kContactSourceWeights])
                                                          : contactAt(b, c, src, p.ipcActivation);
                if (!source.valid) {
                  geomFinite = false;
                  continue;
                }
                uint32_t ctype;
                const uint4 cq = contactIndices(b, c, &ctype);
                if (ipcWeightFor(cq, make_float4(1.f, 1.f, 1.f, 1.f), v) == 0.0f) continue;
                const bool nearMinimum = !(source.distance - dl > p.ipcMinDistance);
                const bool mayChange = source.distance - dl < p.ipcActivation;
                const bool friction = p.ipcFriction > 0.0f && cst[kContactLagged].w > 0.0f;
                ContactData trial = {p.ipcActivation, f3(1, 0, 0), make_float4(0, 0, 0, 0), true};
                if (nearMinimum || mayChange) trial = contactAt(b, c, src, p.ipcActivation, v, trialPos);
                if (nearMinimum) {
                  if (!trial.valid) geomFinite = false;
                  else if (!(trial.distance > p.ipcMinDistance)) jmin = fminf(jmin, 0.0f);
                }
                if (mayChange || friction)
                  de += contactEnergy(b, p, c, trial, src, v, trialPos) -
                        contactEnergy(b, p, c, source, src, 0xffffffffu, f3(0, 0, 0));
              }
            }
            jmin = groupMin<W>(jmin, mask);
            const bool allFinite = __all_sync(mask, geomFinite);
            de = groupSum<W>(de, mask);
            if (!allFinite) { status = kNonfinite; minTrialDet = 0.f; backtracks = bt; break; }
            const float trialMin = fminf(controlMin, jmin);
            minTrialDet = trialMin;
            if (trialMin > kDeterminantFloor) {
              de += inertia * (dot3(position - predV, td) + 0.5f * dot3(td, td)) + floorDelta(p, position.y, td.y);
              if (objActive) de += objectiveDelta(p, b, v, position, td);
              evals += 1;
              if (!finiteS(de)) { status = kNonfinite; backtracks = bt; break; }
              const float tb = kArmijoC1 * gd;
              if (de <= tb) {
                alpha = ta; acceptedDelta = de; bound = tb; backtracks = bt; status = kAccepted;
                acceptedD = td; acceptedP = tp;
                break;
              }
            }
            ta *= kBacktrackFactor;
          }
          if (status == kLineSearchFailed) backtracks = kMaxBacktracks;
        }
        if (lane == 0) {
          tgt[v] = make_float4(acceptedP.x, acceptedP.y, acceptedP.z, 1.0f);
          b.finalUpdate[v] = scaledLength(acceptedD);
          float4* L = &b.local[4ull * v];
          const float4 l0 = make_float4(dr.direction.x, dr.direction.y, dr.direction.z, alpha);
          const float4 l1 = make_float4(dr.minEig * dr.scale, dr.scale, dr.shift * dr.scale, dr.shift);
          const float4 l2 = make_float4(acceptedDelta, bound, dr.gdd, dr.residual);
          const float4 l3 = make_float4(minTrialDet, float(backtracks), float(evals), float(status));
          L[0] = l0; L[1] = l1; L[2] = l2; L[3] = l3;
          localValid = finiteS(l0.x) && finiteS(l0.y) && finiteS(l0.z) && finiteS(l0.w) && finiteS(l1.x) &&
                       finiteS(l1.y) && finiteS(l1.z) && finiteS(l1.w) && finiteS(l2.x) && finiteS(l2.y) &&
                       finiteS(l2.z) && finiteS(l2.w) && finiteS(l3.x) && status != kNonfinite && l1.w >= 0.0f;
          shiftN = dr.shift;
          haveRecord = true;
        }
      }
    }
  }
  // Local aggregates of reduceCandidate's vertex loop (jgs2-shader.ts:3689-3790),
  // per scene: folded in shared memory when the block's vertices share one
  // scene, otherwise added per vertex.
  const bool oneScene = __syncthreads_and(!haveVertex || scene == sScene) != 0;
  if (haveRecord && lane == 0) {
    const bool failure = status == kShiftLimit || status == kNonDescent || status == kLineSearchFailed ||
                         status == kNonfinite || status == kCholeskyFailed;
    uint32_t trials = 0;
    if (status == kAccepted) trials = backtracks + 1;
    else if (status == kLineSearchFailed && backtracks == kMaxBacktracks) trials = kTrialCount;
    else if (status == kZeroGradient && backtracks > 0) trials = backtracks;
    else if (status == kNonfinite) trials = backtracks;  // a nonfinite trial never has J above the floor here
    const uint32_t skipped = trials - (trials < evals ? trials : evals);
    const uint32_t shiftBits = (shiftN > 0.0f && finiteS(shiftN)) ? __float_as_uint(shiftN) : 0u;
    if (oneScene) {
      if (failure) atomicAdd(&sFail, 1u);
      if (backtracks) atomicMax(&sMaxBack, backtracks);
      if (skipped) atomicAdd(&sSkip, skipped);
      if (evals) atomicAdd(&sEvals, evals);
      if (shiftBits) atomicMax(&sMaxShift, shiftBits);
      if (!localValid) sValid = 0;
    } else {
      FrameState* fs = &b.frames[scene];
      if (failure) atomicAdd(&fs->localFailures, 1u);
      if (backtracks) atomicMax(&fs->localMaxBacktracks, backtracks);
      if (skipped) atomicAdd(&fs->localSkipped, skipped);
      if (evals) atomicAdd(&fs->localEvaluations, evals);
      if (shiftBits) atomicMax(&fs->localMaxShift, shiftBits);
      if (!localValid) atomicAnd(&fs->localNumericsValid, 0u);
    }
  }
  __syncthreads();
  if (oneScene && threadIdx.x == 0) {
    FrameState* fs = &b.frames[sScene];
    if (sFail) atomicAdd(&fs->localFailures, sFail);
    if (sMaxBack) atomicMax(&fs->localMaxBacktracks, sMaxBack);
    if (sSkip) atomicAdd(&fs->localSkipped, sSkip);
    if (sEvals) atomicAdd(&fs->localEvaluations, sEvals);
    if (sMaxShift) atomicMax(&fs->localMaxShift, sMaxShift);
    if (!sValid) atomicAnd(&fs->localNumericsValid, 0u);
  }
}

// kCache: the records' line-search state is cached in shared memory (and the
// records are staged there); wide records (an exact complement) recompute it
// per trial instead, so a block needs no shared memory per vertex.
template <int W, bool kExt, bool kCache>
__global__ void __launch_bounds__(kBlock, JGS2_SOLVE_MIN_BLOCKS) solveKernel(Buffers b, const DevParams* __restrict__ pp,
                                                      const float4* __restrict__ src, float4* tgt,
                                                      const uint32_t* __restrict__ list, uint32_t count,
                                                      uint32_t K, int cachedIncident, uint32_t groupsPerBlock) {
  solveChunk<W, kExt, false, kCache>(b, pp, src, tgt, list, count, K, cachedIncident, groupsPerBlock, blockIdx.x);
}

// ---------------------------------------------------------------------------
// The same local solve with the block's work spread over its threads by item
// instead of by vertex: solid scenes (no cloth, no contact) whose records fit
// shared memory.  A block takes up to kG vertices and goes through
//   records   one thread per cubature record: its state to shared memory, its
//             gradient and Hessian contribution to a row;
//   incident  (coloured sweeps) one thread per incident tet, likewise;
//   sums      four lanes per vertex add the rows in solveChunk's order;
//   solve     one thread per vertex: globalization and the line search's
//             bookkeeping;
//   trial     per line-search trial one thread per record and per incident tet
//             evaluates its energy delta and determinant, and four lanes per
//             vertex add them.
// A record's or tet's arithmetic and the order of every sum are solveChunk's,
// so a vertex takes the same step, bit for bit, in either kernel and for any
// kG (the recorded energy delta of an accepted trial can differ in its last
// bit).
//
// Bound by latency: with few vertices a launch is one block's chain of
// phases.  solveChunk's chain is two passes of four lanes over six records,
// six passes over 24 incident tets per trial and up to 13 trials; here a
// record or tet is one pass and, at eight vertices a block, a thread keeps its
// incident tet's deformation gradient over the trials and six backtracked
// trials are evaluated at a time: a vertex that goes through all thirteen takes
// three rounds, and six is what four summing lanes each leave room for (sweeps
// of a colour-locked 525-vertex bar 4.99 ms two at a time, 4.36 four, 4.23
// six; of a 27 360-vertex block 5.48, 4.98, 4.87).  Measured per launch (events; four lanes,
// then items): 525 vertices 27.0 / 18.9 us, 2 688 vertices 35 / 27, 13 392
// vertices 44.6 / 39.4; one colour of the 525-vertex bar, whose trials a
// determinant bound often holds back, 72 / 33, of a 27 360-vertex block
// 85 / 36.  A large solve is better off with four lanes (1 030 301 vertices:
// 1.72 ms, 1.79 by items, 68 921: 139 / 142 us): both run out of warps to hide
// the gathers behind, and the block's barriers then cost more than the idle
// lanes.
constexpr uint32_t kItemTrials = 6;   // backtracked trials evaluated at a time
constexpr uint32_t kItemTets = 24;    // incident tets of a vertex per round (the grid meshes' largest valence)
constexpr uint32_t kBasisWords = 9;   // float4 per record: basis blocks, then dF (27), gQ (3), HQ (6)
constexpr uint32_t kStateWords = 5;   // float4 per record: F, vol, lambda, mu, gs, w, I0, J0, slot; an odd stride
constexpr uint32_t kRowFloats = 18;   // floats per record row: w R_s g (3), R_s H R_s^T (6), own block (3 + 6)
constexpr uint32_t kTetRowFloats = 10;  // floats per incident row: gradient (3), Hessian block (6), vol

__host__ __device__ constexpr uint32_t itemScratchFloats(uint32_t groups, uint32_t K, bool incident, uint32_t trials) {
  const uint32_t gather = groups * (K * kRowFloats + (incident ? kItemTets * kTetRowFloats : 0u));
  const uint32_t trial = trials * groups * (K * 2u + kItemTets * 3u);
  return ((gather > trial ? gather : trial) + 3u) & ~3u;
}
__host__ __device__ constexpr size_t itemSharedBytes(uint32_t groups, uint32_t K, bool incident, uint32_t trials) {
  return size_t(groups) * K * (kBasisWords + kStateWords) * 16 +
         size_t(itemScratchFloats(groups, K, incident, trials)) * 4;
}

template <uint32_t kG, uint32_t kT>
struct ItemShared {
  uint32_t v[kG], scene[kG], start[kG], count[kG];
  uint32_t solve[kG];            // the vertex takes a local solve
  uint32_t eval[kG];             // trials of it to evaluate this round
  // Per trial of the round: the step, the step in the vertex's frame and the
  // terms a record at the vertex's own slot takes out.
  float td[kT][kG][3], ts[kT][kG][3], ownMove[kT][kG], ownObjective[kT][kG];
  float sum[kG][12];             // gradient, its compensation, Hessian
  float4 own[kG][6];             // staged: source pose, target, rest and mass, incident system
  float de[kT][kG], jmin[kT][kG];
  uint32_t finite[kT][kG];
  uint32_t fail, maxBack, skip, evals, maxShift, valid;
};

// An incident tet's terms with every fused multiply-add spelled out (the first
// product fused onto the second, as the compiler contracts the plain
// expressions of solveChunk): the coloured sweep amplifies a last bit to whole
// steps, and the compiler contracts differently once the deformation gradient
// is kept across phases.
namespace fused {
__device__ __forceinline__ float sum2(float a, float x, float b, float y) { return __fmaf_rn(a, x, __fmul_rn(b, y)); }
__device__ __forceinline__ float diff2(float a, float x, float b, float y) { return __fmaf_rn(a, x, -__fmul_rn(b, y)); }
__device__ __forceinline__ float dot(float3 a, float3 b) { return __fmaf_rn(a.z, b.z, sum2(a.x, b.x, a.y, b.y)); }
__device__ __forceinline__ float3 cross(float3 a, float3 b) {
  return f3(diff2(a.y, b.z, a.z, b.y), diff2(a.z, b.x, a.x, b.z), diff2(a.x, b.y, a.y, b.x));
}
// a x + b y + c z, column by column.
__device__ __forceinline__ float3 combine(float3 a, float x, float3 b, float y, float3 c, float z) {
  return f3(__fmaf_rn(c.x, z, sum2(a.x, x, b.x, y)), __fmaf_rn(c.y, z, sum2(a.y, x, b.y, y)),
            __fmaf_rn(c.z, z, sum2(a.z, x, b.z, y)));
}
__device__ __forceinline__ float3 timesF(const M3& m, float3 v) { return combine(m.c0, v.x, m.c1, v.y, m.c2, v.z); }
__device__ __forceinline__ M3 cofactorF(const M3& f) { return {cross(f.c1, f.c2), cross(f.c2, f.c0), cross(f.c0, f.c1)}; }
__device__ __forceinline__ float det(const M3& f) { return dot(f.c0, cross(f.c1, f.c2)); }
__device__ __forceinline__ float squared(const M3& f) {
  return __fadd_rn(__fadd_rn(dot(f.c0, f.c0), dot(f.c1, f.c1)), dot(f.c2, f.c2));
}
__device__ __forceinline__ M3 deformation(const TetRec& r, const float4* __restrict__ x) {
  const float3 o = xyz(x[r.idx.x]);
  const float3 a = xyz(x[r.idx.y]) - o, b = xyz(x[r.idx.z]) - o, c = xyz(x[r.idx.w]) - o;
  return {combine(a, r.g1.x, b, r.g2.x, c, r.g3.x), combine(a, r.g1.y, b, r.g2.y, c, r.g3.y),
          combine(a, r.g1.z, b, r.g2.z, c, r.g3.z)};
}

// Gradient vol P g and Hessian block (without vol) of the tet's vertex with
// shape gradient g (piolaTerms, piola, incidentBlock).
__device__ __forceinline__ void incident(const M3& F, float3 g, float vol, float lambda, float mu, float3* grad,
                                         S3* block) {
  const float den = squared(F) + 1.0f;
  const M3 cof = cofactorF(F);
  const float J = dot(F.c0, cof.c0);
  const float a = __fmul_rn(mu, 1.0f - 1.0f / den);
  const float b = diff2(lambda, J - 1.0f, 0.75f, mu);
  const float c1 = __fmul_rn(2.0f, mu) / __fmul_rn(den, den);
  auto stress = [&](float3 f, float3 c) { return f3(sum2(a, f.x, b, c.x), sum2(a, f.y, b, c.y), sum2(a, f.z, b, c.z)); };
  const M3 P = {stress(F.c0, cof.c0), stress(F.c1, cof.c1), stress(F.c2, cof.c2)};
  const float3 Pg = timesF(P, g), u = timesF(F, g), w = timesF(cof, g);
  *grad = f3(__fmul_rn(vol, Pg.x), __fmul_rn(vol, Pg.y), __fmul_rn(vol, Pg.z));
  const float d = __fmul_rn(a, dot(g, g));
  auto entry = [&](float diagonal, float u0, float u1, float w0, float w1) {
    return __fmaf_rn(__fmul_rn(lambda, w0), w1, __fmaf_rn(__fmul_rn(c1, u0), u1, diagonal));
  };
  *block = {entry(d, u.x, u.x, w.x, w.x),    entry(d, u.y, u.y, w.y, w.y),    entry(d, u.z, u.z, w.z, w.z),
            entry(0.0f, u.x, u.y, w.x, w.y), entry(0.0f, u.x, u.z, w.x, w.z), entry(0.0f, u.y, u.z, w.y, w.z)};
}

// snhEnergyDeltaRankOne of a step d of that vertex.
__device__ __forceinline__ float energyDelta(const M3& F, float3 d, float3 g, float lambda, float mu, float* Jtrial) {
  const float I0 = squared(F), J0 = det(F);
  const float id = __fmaf_rn(dot(d, d), dot(g, g), __fmul_rn(2.0f, dot(d, timesF(F, g))));
  const float dj = dot(d, timesF(cofactorF(F), g));
  auto moved = [&](float3 c, float s) { return f3(__fmaf_rn(d.x, s, c.x), __fmaf_rn(d.y, s, c.y), __fmaf_rn(d.z, s, c.z)); };
  const M3 f1 = {moved(F.c0, g.x), moved(F.c1, g.y), moved(F.c2, g.z)};
  const float J1 = det(f1);
  *Jtrial = J1;
  const float lr = logOnePlus(id / (I0 + 1.0f));
  const float half = __fmul_rn(0.5f, mu);
  float e = diff2(half, id, __fmul_rn(0.75f, mu), dj);
  e = __fmaf_rn(__fmul_rn(__fmul_rn(0.5f, lambda), dj), J1 + J0 - 2.0f, e);
  return __fmaf_rn(-half, lr, e);
}
}  // namespace fused

template <uint32_t kG, uint32_t kItemThreads, bool kJacobi, int kMinBlocks>
__global__ void __launch_bounds__(kItemThreads, kMinBlocks)
    solveItemsKernel(Buffers b, const DevParams* __restrict__ pp, const float4* __restrict__ src, float4* tgt,
                     const uint32_t* __restrict__ list, uint32_t count, uint32_t K, uint32_t groups) {
  extern __shared__ float4 cache4[];
  // One incident tet per thread and round, kept over the trials; then also
  // kTrials backtracked trials at a time once the first one has failed.
  constexpr bool kHold = kG * kItemTets == kItemThreads;
  constexpr uint32_t kTrials = kHold ? kItemTrials : 1u;
  __shared__ ItemShared<kG, kTrials> sh;
  float4* basisS = cache4;
  float4* stateS = cache4 + size_t(groups) * K * kBasisWords;
  float* rows = reinterpret_cast<float*>(stateS + size_t(groups) * K * kStateWords);
  float* tetRows = rows + groups * K * kRowFloats;
  const uint32_t tid = threadIdx.x;
  const uint32_t first = blockIdx.x * groups, n = min(groups, count - first);
  const uint32_t nrec = n * K;

  // ---- vertices: what the block's threads need of each, and the ones that
  // take no solve (jgs2-shader.ts:3042-3081 for the preflight rejection) ----
  uint32_t status = kNonfinite, backtracks = 0, evals = 0;
  float shiftN = 0.0f;
  bool localValid = true, haveRecord = false;
  if (tid == kItemThreads - 1) {
    sh.fail = sh.maxBack = sh.skip = sh.evals = sh.maxShift = 0u;
    sh.valid = 1u;
  }
  if (tid < groups) {
    uint32_t solve = 0, v = 0, scene = 0;
    bool have = tid < n;
    if (have) v = list ? list[first + tid] : first + tid;
    have = have && inBounds(v, b.vertexTotal, kSiteListVertex);
    sh.count[tid] = 0u;
    if (have) {
      scene = b.vertexScene[v];
      const DevParams& p = pp[scene];
      if (p.active) {
        const FrameState* fs = &b.frames[scene];
        const uint4 info = b.vinfo[v];
        sh.start[tid] = info.x;
        sh.count[tid] = info.y;
        if (latched(p, fs)) {
          tgt[v] = src[v];
        } else if (isPinned(info)) {
          const float4 rm = b.restMass[v];
          tgt[v] = make_float4(rm.x, rm.y, rm.z, 1.0f);
          b.finalUpdate[v] = 0.0f;
          float4* L = &b.local[4ull * v];
          L[0] = L[1] = L[2] = make_float4(0, 0, 0, 0);
          L[3] = make_float4(0, 0, 0, float(kPinned));
          status = kPinned;
          haveRecord = true;
        } else {
          const float4 c0 = fs->control[0];
          const uint32_t vb = controlBits(c0.w) & kValidityMask;
          const bool amv = (vb & kAcceptedMinimumValid) != 0u && finiteS(c0.z);
          if (!(amv && c0.z > kDeterminantFloor)) {
            tgt[v] = src[v];
            b.finalUpdate[v] = 0.0f;
            float4* L = &b.local[4ull * v];
            L[0] = L[1] = L[2] = make_float4(0, 0, 0, 0);
            status = amv ? kLineSearchFailed : kNonfinite;
            L[3] = make_float4(amv ? c0.z : 0.f, 0, 0, float(status));
            localValid = status != kNonfinite;
            haveRecord = true;
          } else {
            solve = 1;
          }
        }
      }
    }
    sh.v[tid] = v;
    sh.scene[tid] = scene;
    sh.solve[tid] = solve;
  }
  // ---- basis blocks: staged as they lie, sixteen bytes a copy ----
  if (list == nullptr) {
    const float4* from = b.cubBasis + size_t(first) * K * kBasisWords;
    for (uint32_t c = tid; c < nrec * kBasisWords; c += kItemThreads) cpAsync16(&basisS[c], from + c);
  } else {
    const uint32_t per = K * kBasisWords;
    for (uint32_t c = tid; c < n * per; c += kItemThreads) {
      const uint32_t g = c / per, v = list[first + g];
      if (inBounds(v, b.vertexTotal, kSiteListVertex)) cpAsync16(&basisS[c], b.cubBasis + size_t(v) * per + (c - g * per));
    }
  }
  // The vertex's own data, wanted by one thread per vertex only later, when
  // nothing else of the block would hide its latency.
  for (uint32_t c = tid; c < n * 6u; c += kItemThreads) {
    const uint32_t g = c / 6u, part = c - g * 6u, w = list ? list[first + g] : first + g;
    if (!inBounds(w, b.vertexTotal, kSiteListVertex)) continue;
    if (part == 0u) cpAsync16(&sh.own[g][0], src + w);
    else if (part == 1u) cpAsync16(&sh.own[g][1], b.predicted + w);
    else if (part == 2u) cpAsync16(&sh.own[g][2], b.restMass + w);
    else if (kJacobi) cpAsync16(&sh.own[g][part], b.incident + 3ull * w + (part - 3u));
  }
  cpAsyncWaitAll();
  __syncthreads();

  // ---- records (jgs2-shader.ts:3197-3263) ----
  for (uint32_t i = tid; i < nrec; i += kItemThreads) {
    const uint32_t g = i / K;
    if (!sh.solve[g]) continue;
    const uint32_t v = sh.v[g];
    const DevParams& p = pp[sh.scene[g]];
    const bool objActive = p.objectiveFlags != 0u;
    const size_t rec = size_t(v) * K + (i - g * K);
    const uint4 head = __ldg(&b.cubHead[2 * rec]), idx = __ldg(&b.cubHead[2 * rec + 1]);
    const float w = __uint_as_float(head.y);
    float4* state = stateS + i * kStateWords;
    if (!(head.x != kEmptyTet && w > 0.0f) || !inBounds(head.x, b.tetTotal, kSiteRecordTet) ||
        !inBounds(idx.x, b.vertexTotal, kSiteRecordVertex) || !inBounds(idx.y, b.vertexTotal, kSiteRecordVertex) ||
        !inBounds(idx.z, b.vertexTotal, kSiteRecordVertex) || !inBounds(idx.w, b.vertexTotal, kSiteRecordVertex)) {
      state[3].w = 0.0f;
      continue;
    }
    const TetRec r = loadTet(b.tets, head.x);
    const M3 Rs = loadFrame(b.vertexPack, v);
    CubState st;
    recordStateOf<false>(b, p, v, w, idx, r, [&](int l) { return loadBlockVecShared(basisS + i * kBasisWords, l); },
                         src, objActive, st);
    const M3& F = st.F;
    const M3 &dF0 = st.dF0, &dF1 = st.dF1, &dF2 = st.dF2;
    const PiolaTerms pt = piolaTerms(F, r.lambda, r.mu);
    const M3 P = piola(F, pt);
    const float3 pg = r.vol * f3(frob(dF0, P), frob(dF1, P), frob(dF2, P)) + st.gQ;
    const float p0 = frob(F, dF0), p1 = frob(F, dF1), p2 = frob(F, dF2);
    const float q0 = frob(pt.cof, dF0), q1 = frob(pt.cof, dF1), q2 = frob(pt.cof, dF2);
    S3 ph;
    {
      const M3 D0 = dcofactor(F, dF0);
      ph.xx = pt.b * frob(dF0, D0);
      ph.xy = pt.b * frob(dF1, D0);
      ph.xz = pt.b * frob(dF2, D0);
    }
    {
      const M3 D1 = dcofactor(F, dF1);
      ph.yy = pt.b * frob(dF1, D1);
      ph.yz = pt.b * frob(dF2, D1);
    }
    ph.zz = pt.b * frob(dF2, dcofactor(F, dF2));
    ph.xx += pt.a * frob(dF0, dF0) + pt.c1 * p0 * p0 + r.lambda * q0 * q0;
    ph.yy += pt.a * frob(dF1, dF1) + pt.c1 * p1 * p1 + r.lambda * q1 * q1;
    ph.zz += pt.a * frob(dF2, dF2) + pt.c1 * p2 * p2 + r.lambda * q2 * q2;
    ph.xy += pt.a * frob(dF0, dF1) + pt.c1 * p0 * p1 + r.lambda * q0 * q1;
    ph.xz += pt.a * frob(dF0, dF2) + pt.c1 * p0 * p2 + r.lambda * q0 * q2;
    ph.yz += pt.a * frob(dF1, dF2) + pt.c1 * p1 * p2 + r.lambda * q1 * q2;
    ph.xx *= r.vol; ph.yy *= r.vol; ph.zz *= r.vol; ph.xy *= r.vol; ph.xz *= r.vol; ph.yz *= r.vol;
    sadd(ph, st.HQ);
    const float3 wg = w * mv(Rs, pg);
    const S3 wh = srotate(Rs, ph);
    float* row = rows + i * kRowFloats;
    row[0] = wg.x; row[1] = wg.y; row[2] = wg.z;
    row[3] = wh.xx; row[4] = wh.yy; row[5] = wh.zz; row[6] = wh.xy; row[7] = wh.xz; row[8] = wh.yz;
    if (st.slot < 4) {
      // The exact source block already in the local gather.
      const float3 position = xyz(src[v]);
      const float4 pv = b.predicted[v];
      const float3 gs = st.gs;
      // The fused forms solveChunk compiles to, spelled out.
      const float3 away = position - xyz(pv), stress = mv(P, gs);
      float3 ps = f3(__fmaf_rn(pv.w, away.x, __fmul_rn(r.vol, stress.x)),
                     __fmaf_rn(pv.w, away.y, __fmul_rn(r.vol, stress.y)),
                     __fmaf_rn(pv.w, away.z, __fmul_rn(r.vol, stress.z)));
      if (objActive) {
        const float share = 1.0f / float(sh.count[g] > 1u ? sh.count[g] : 1u);
        const float3 og = objectiveGradient(p, b, v, position);
        ps = f3(__fadd_rn(ps.x, __fmul_rn(og.x, share)), __fadd_rn(ps.y, __fmul_rn(og.y, share)),
                __fadd_rn(ps.z, __fmul_rn(og.z, share)));
      }
      const S3 blk = incidentBlock(r, F, pt, gs);
      const float3 wp = (-w) * ps;
      row[9] = wp.x; row[10] = wp.y; row[11] = wp.z;
      row[12] = blk.xx; row[13] = blk.yy; row[14] = blk.zz; row[15] = blk.xy; row[16] = blk.xz; row[17] = blk.yz;
    }
    // The state the trials read, over the basis it was formed from.
    state[0] = make_float4(F.c0.x, F.c0.y, F.c0.z, r.vol);
    state[1] = make_float4(F.c1.x, F.c1.y, F.c1.z, r.lambda);
    state[2] = make_float4(F.c2.x, F.c2.y, F.c2.z, r.mu);
    state[3] = make_float4(st.gs.x, st.gs.y, st.gs.z, w);
    state[4] = make_float4(st.I0, st.J0, __uint_as_float(st.slot), 0.0f);
    float4* d = basisS + i * kBasisWords;
    d[0] = make_float4(dF0.c0.x, dF0.c0.y, dF0.c0.z, dF0.c1.x);
    d[1] = make_float4(dF0.c1.y, dF0.c1.z, dF0.c2.x, dF0.c2.y);
    d[2] = make_float4(dF0.c2.z, dF1.c0.x, dF1.c0.y, dF1.c0.z);
    d[3] = make_float4(dF1.c1.x, dF1.c1.y, dF1.c1.z, dF1.c2.x);
    d[4] = make_float4(dF1.c2.y, dF1.c2.z, dF2.c0.x, dF2.c0.y);
    d[5] = make_float4(dF2.c0.z, dF2.c1.x, dF2.c1.y, dF2.c1.z);
    d[6] = make_float4(dF2.c2.x, dF2.c2.y, dF2.c2.z, st.gQ.x);
    d[7] = make_float4(st.gQ.y, st.gQ.z, st.HQ.xx, st.HQ.yy);
    d[8] = make_float4(st.HQ.zz, st.HQ.xy, st.HQ.xz, st.HQ.yz);
  }

  // ---- incident tets ----
  uint32_t most = 0;
  for (uint32_t g = 0; g < n; ++g) most = max(most, sh.solve[g] ? sh.count[g] : 0u);
  struct HeldTet {
    M3 F;
    float3 g;
    float vol, lambda, mu;
    bool ok;
  };
  auto loadHeld = [&](uint32_t g, uint32_t a, HeldTet& h) {
    h.ok = false;
    if (g >= n || !sh.solve[g] || a >= sh.count[g]) return;
    const uint32_t entry = __ldg(&b.adjacency[sh.start[g] + a]);
    TetRec r;
    if (!incidentTetChecked(b.tets, entry, b.tetTotal, b.vertexTotal, &r)) return;
    h.F = fused::deformation(r, src);
    h.g = shapeGradient(r, entry & 3u);
    h.vol = r.vol; h.lambda = r.lambda; h.mu = r.mu;
    h.ok = true;
  };
  HeldTet held;
  held.ok = false;
  if constexpr (kHold) loadHeld(tid / kItemTets, tid % kItemTets, held);
  // ---- sums: lane j of a vertex's four takes records j, j + 4, ... and
  // (coloured sweeps) incident tets j, j + 4, ... ----
  const uint32_t sg = tid / 4, lane = tid & 3u;
  const unsigned mask = 0xfu << (tid & 28u);
  const bool summing = sg < n && sh.solve[sg] != 0u;
  Comp3 gsum = czero();
  S3 hess = szero();
  // A checked build may reject a tet that the sums go over: its terms are none.
  constexpr bool kRejects = JGS2_BOUNDS_CHECKS != 0;
  auto incidentRow = [&](uint32_t i, const HeldTet& h) {
    if (!h.ok) {
      if (kRejects)
        for (uint32_t k = 0; k < kTetRowFloats; ++k) tetRows[i * kTetRowFloats + k] = 0.0f;
      return;
    }
    float3 f;
    S3 blk;
    fused::incident(h.F, h.g, h.vol, h.lambda, h.mu, &f, &blk);
    float* row = tetRows + i * kTetRowFloats;
    row[0] = f.x; row[1] = f.y; row[2] = f.z;
    row[3] = blk.xx; row[4] = blk.yy; row[5] = blk.zz; row[6] = blk.xy; row[7] = blk.xz; row[8] = blk.yz;
    row[9] = h.vol;
  };
  auto incidentRound = [&](uint32_t a0) {
    for (uint32_t i = tid; i < n * kItemTets; i += kItemThreads) {
      HeldTet h;
      if (kHold && a0 == 0) h = held;
      else loadHeld(i / kItemTets, a0 + i % kItemTets, h);
      incidentRow(i, h);
    }
  };
  if constexpr (!kJacobi) incidentRound(0);
  __syncthreads();
  if (summing) {
    const uint32_t v = sh.v[sg];
    for (uint32_t u = lane; u < K; u += 4) {
      const float* row = rows + (sg * K + u) * kRowFloats;
      const float4* state = stateS + (sg * K + u) * kStateWords;
      const float w = state[3].w;
      if (!(w > 0.0f)) continue;
      cadd(gsum, f3(row[0], row[1], row[2]));
      saddScaled(hess, w, S3{row[3], row[4], row[5], row[6], row[7], row[8]});
      if (__float_as_uint(state[4].z) < 4u) {
        const DevParams& p = pp[sh.scene[sg]];
        const float nS = float(sh.count[sg] > 1u ? sh.count[sg] : 1u);
        cadd(gsum, f3(row[9], row[10], row[11]));
        saddScaled(hess, -w * state[0].w, S3{row[12], row[13], row[14], row[15], row[16], row[17]});
        const float own = b.predicted[v].w + targetStiffness(p, b, v) / nS;
        hess.xx = __fmaf_rn(-w, own, hess.xx);
        hess.yy = __fmaf_rn(-w, own, hess.yy);
        hess.zz = __fmaf_rn(-w, own, hess.zz);
      }
    }
  }
  if constexpr (!kJacobi) {
    for (uint32_t a0 = 0; a0 == 0 || a0 < most; a0 += kItemTets) {
      if (a0 > 0) {
        __syncthreads();
        incidentRound(a0);
        __syncthreads();
      }
      if (summing)
        for (uint32_t j = lane; j < kItemTets && a0 + j < sh.count[sg]; j += 4) {
          const float* row = tetRows + (sg * kItemTets + j) * kTetRowFloats;
          cadd(gsum, f3(row[0], row[1], row[2]));
          saddScaled(hess, row[9], S3{row[3], row[4], row[5], row[6], row[7], row[8]});
        }
    }
  }
  if (summing) {
    groupMerge<4>(gsum, mask);
    hess.xx = groupSum<4>(hess.xx, mask);
    hess.yy = groupSum<4>(hess.yy, mask);
    hess.zz = groupSum<4>(hess.zz, mask);
    hess.xy = groupSum<4>(hess.xy, mask);
    hess.xz = groupSum<4>(hess.xz, mask);
    hess.yz = groupSum<4>(hess.yz, mask);
    if (lane == 0) {
      float* o = sh.sum[sg];
      o[0] = gsum.s.x; o[1] = gsum.s.y; o[2] = gsum.s.z;
      o[3] = gsum.c.x; o[4] = gsum.c.y; o[5] = gsum.c.z;
      o[6] = hess.xx; o[7] = hess.yy; o[8] = hess.zz; o[9] = hess.xy; o[10] = hess.xz; o[11] = hess.yz;
    }
  }
  __syncthreads();

  // ---- globalization (jgs2-shader.ts:3265-3473), one thread per vertex ----
  const bool solving = tid < n && sh.solve[tid] != 0u;
  const uint32_t v = tid < n ? sh.v[tid] : 0u;
  const DevParams& p = pp[tid < n ? sh.scene[tid] : 0u];
  SolveResult dr{f3(0, 0, 0), 0, 0, 0, 0, 0, kNonfinite};
  float3 position = f3(0, 0, 0), predV = f3(0, 0, 0), grad = f3(0, 0, 0);
  float inertia = 0.0f, resolution = 0.0f, controlMin = 0.0f;
  float alpha = 0.0f, acceptedDelta = 0.0f, bound = 0.0f, minTrialDet = 0.0f, ta = 1.0f;
  float3 acceptedD = f3(0, 0, 0), acceptedP = f3(0, 0, 0);
  uint32_t bt = 0;
  bool searching = false;
  if (solving) {
    position = xyz(sh.own[tid][0]);
    predV = xyz(sh.own[tid][1]);
    acceptedP = position;
    inertia = sh.own[tid][2].w * p.invDt2;
    const bool objActive = p.objectiveFlags != 0u;
    const float3 objS = objActive ? objectiveGradient(p, b, v, position) : f3(0, 0, 0);
    const float* o = sh.sum[tid];
    Comp3 gs;
    gs.s = f3(o[0], o[1], o[2]);
    gs.c = f3(o[3], o[4], o[5]);
    S3 h = {o[6], o[7], o[8], o[9], o[10], o[11]};
    if constexpr (kJacobi) {
      const float4 i0 = sh.own[tid][3], i1 = sh.own[tid][4], i2 = sh.own[tid][5];
      cadd(gs, f3(i0.x, i0.y, i0.z));
      h.xx += i0.w;
      h.yy += i1.x;
      h.zz += i1.y;
      h.xy += i1.z;
      h.xz += i1.w;
      h.yz += i2.x;
    }
    // Own terms: inertia, objectives, floor (jgs2-shader.ts:3083-3092, 3188-3191).
    cadd(gs, inertia * (position - predV));
    saddDiag(h, inertia);
    if (objActive) cadd(gs, objS);
    if (p.objectiveFlags & 2u) saddDiag(h, targetStiffness(p, b, v));
    if (p.floorStiffness > 0.0f && position.y < p.floorHeight) {
      cadd(gs, f3(0.0f, p.floorStiffness * (position.y - p.floorHeight), 0.0f));
      h.yy += p.floorStiffness;
    }
    grad = cvalue(gs);
    dr = globalizationSolve(h, grad, inertia);
    status = kNonfinite;
    const float3 fullP = position + dr.direction;
    const float3 fullD = fullP - position;
    const float scs = fmaxf(fabsf(position.x), fmaxf(fabsf(position.y), fabsf(position.z)));
    resolution = fmaxf(p.sceneScale, fmaxf(scs, 1.0e-12f)) * kUnitRoundoff * kPositionResolutionMultiplier;
    const bool below = dr.status == kAccepted && finiteV(fullP) && finiteV(fullD) && scaledLength(fullD) <= resolution;
    if (dr.status == kAccepted) status = below ? kZeroGradient : kLineSearchFailed;
    else if (dr.status == kZeroGradient) status = kZeroGradient;
    else if (dr.status == kShiftLimit) status = kShiftLimit;
    else if (dr.status == kCholeskyFailed) status = kCholeskyFailed;
    else if (dr.status == kNonDescent) status = kNonDescent;
    if (dr.status == kAccepted && !below) {
      searching = true;
      const float dl = scaledLength(dr.direction);
      if (p.maxStep > 0.0f && dl > p.maxStep) ta = p.maxStep / dl;
      controlMin = b.frames[sh.scene[tid]].control[0].z;  // accepted-source minimum (finite here)
    }
  }
  // ---- line search ----
  // A round evaluates the first trial alone and then, where a thread holds its
  // incident tet, the next kTrials of the backtracking sequence together: they
  // do not depend on one another, and a vertex that a determinant bound holds
  // back goes through all thirteen.  The trials are then judged in order.
  uint32_t roundTrials = 1u;
  for (;;) {
    uint32_t evalCount = 0, firstBt = bt;
    float firstTa = ta;
    if (searching) {
      searching = false;
      for (; bt <= kMaxBacktracks; ++bt) {
        const float3 tp = position + ta * dr.direction;
        const float3 td = tp - position;
        if (!finiteV(tp) || !finiteV(td)) {
          if (evalCount == 0) { status = kNonfinite; minTrialDet = 0.f; backtracks = bt; }
          break;
        }
        const float tl = scaledLength(td);
        if (p.maxStep > 0.0f && tl > p.maxStep) {
          if (evalCount > 0) break;
          ta *= kBacktrackFactor;
          continue;
        }
        if (tl <= resolution) {
          if (evalCount == 0) { status = kZeroGradient; minTrialDet = 0.f; backtracks = bt; }
          break;
        }
        const float gd = dot3(grad, td);
        if (!finiteS(gd)) {
          if (evalCount == 0) { status = kNonfinite; minTrialDet = 0.f; backtracks = bt; }
          break;
        }
        if (!(gd < 0.0f)) {
          if (evalCount == 0) { status = kZeroGradient; minTrialDet = 0.f; backtracks = bt; }
          break;
        }
        if (evalCount == 0) {
          firstBt = bt;
          firstTa = ta;
        }
        const uint32_t j = evalCount++;
        const float3 ts = mtv(loadFrame(b.vertexPack, v), td);
        sh.td[j][tid][0] = td.x; sh.td[j][tid][1] = td.y; sh.td[j][tid][2] = td.z;
        sh.ts[j][tid][0] = ts.x; sh.ts[j][tid][1] = ts.y; sh.ts[j][tid][2] = ts.z;
        sh.ownMove[j][tid] = dot3(position - predV, td) + 0.5f * dot3(td, td);
        const float nS = float(sh.count[tid] > 1u ? sh.count[tid] : 1u);
        sh.ownObjective[j][tid] = p.objectiveFlags != 0u ? objectiveDelta(p, b, v, position, td) / nS : 0.0f;
        if (evalCount == roundTrials) break;
        ta *= kBacktrackFactor;
      }
    }
    if (tid < groups) sh.eval[tid] = evalCount;
    if (!__syncthreads_or(evalCount != 0u)) break;
    // Restricted geometry and energy (restrictedMinimumDeformationDeterminant
    // :1980-2118 and restrictedEnergyDelta :2120-2337).
    const uint32_t recStride = groups * K * 2u, tetStride = groups * kItemTets * 3u;
    float* recTrial = rows;                                   // (energy, J) per record and trial
    float* tetTrial = rows + roundTrials * recStride;         // (energy, vol, J) per incident tet and trial
    for (uint32_t i = tid; i < nrec * roundTrials; i += kItemThreads) {
      const uint32_t j = kTrials > 1 ? i / nrec : 0u, r = i - j * nrec, g = r / K;
      if (sh.eval[g] <= j) continue;
      const float4* s = stateS + r * kStateWords;
      const float4 s3 = s[3];
      if (!(s3.w > 0.0f)) continue;
      const float4 s0 = s[0], s1 = s[1], s2 = s[2], s4 = s[4];
      const float4* d = basisS + r * kBasisWords;
      const float4 d0 = d[0], d1 = d[1], d2 = d[2], d3 = d[3], d4 = d[4], d5 = d[5], d6 = d[6], d7 = d[7], d8 = d[8];
      const M3 F = {xyz(s0), xyz(s1), xyz(s2)};
      const M3 dF0 = {f3(d0.x, d0.y, d0.z), f3(d0.w, d1.x, d1.y), f3(d1.z, d1.w, d2.x)};
      const M3 dF1 = {f3(d2.y, d2.z, d2.w), f3(d3.x, d3.y, d3.z), f3(d3.w, d4.x, d4.y)};
      const M3 dF2 = {f3(d4.z, d4.w, d5.x), f3(d5.y, d5.z, d5.w), f3(d6.x, d6.y, d6.z)};
      const float3 gQ = f3(d6.w, d7.x, d7.y);
      const S3 HQ = {d7.z, d7.w, d8.x, d8.y, d8.z, d8.w};
      const float vol = s0.w, lambda = s1.w, mu = s2.w;
      const float3 ts = f3(sh.ts[j][g][0], sh.ts[j][g][1], sh.ts[j][g][2]);
      const float3 step = f3(sh.td[j][g][0], sh.td[j][g][1], sh.td[j][g][2]);
      float J = 0.0f;
      // Record state is in the source frame: the trial step there is R_s^T td.
      const M3 D = ts.x * dF0 + ts.y * dF1 + ts.z * dF2;
      const float dm = vol * snhEnergyDelta(F, s4.x, s4.y, D, lambda, mu, &J);
      float comp = dm + dot3(ts, gQ) + 0.5f * dot3(ts, smv(HQ, ts));
      if (__float_as_uint(s4.z) < 4u) {
        float Js;
        comp -= vol * snhEnergyDelta(F, s4.x, s4.y, outer(step, xyz(s3)), lambda, mu, &Js);
        comp -= sh.own[g][1].w * sh.ownMove[j][g];
        if (pp[sh.scene[g]].objectiveFlags != 0u) comp -= sh.ownObjective[j][g];
      }
      recTrial[j * recStride + 2u * r] = comp;
      recTrial[j * recStride + 2u * r + 1u] = J;
    }
    // Four lanes per vertex and trial add its items.
    const uint32_t sj = kTrials > 1 ? sg / n : 0u, av = sg - sj * n;
    const bool adding = sj < roundTrials && sg < n * roundTrials && sh.eval[av] > sj;
    float jmin = kF32Max, de = 0.0f;
    bool geomFinite = true;
    // Lane-order index u >= K of an incident tet is adjacency slot u - K.
    const uint32_t firstInc = lane >= K % 4u ? lane - K % 4u : lane + 4u - K % 4u;
    for (uint32_t a0 = 0; a0 == 0 || a0 < most; a0 += kItemTets) {
      if (a0 > 0) __syncthreads();
      for (uint32_t i = tid; i < n * kItemTets; i += kItemThreads) {
        const uint32_t g = i / kItemTets, trials = sh.eval[g];
        if (trials == 0u) continue;
        HeldTet h;
        if (kHold && a0 == 0) h = held;
        else loadHeld(g, a0 + i % kItemTets, h);
        if (!h.ok) {
          if (kRejects)
            for (uint32_t j = 0; j < trials; ++j) {
              float* t = tetTrial + j * tetStride + 3u * i;
              t[0] = t[1] = 0.0f;
              t[2] = kF32Max;
            }
          continue;
        }
        for (uint32_t j = 0; j < trials; ++j) {
          float J = 0.0f;
          const float e = fused::energyDelta(h.F, f3(sh.td[j][g][0], sh.td[j][g][1], sh.td[j][g][2]), h.g, h.lambda,
                                             h.mu, &J);
          float* t = tetTrial + j * tetStride + 3u * i;
          t[0] = e;
          t[1] = h.vol;
          t[2] = J;
        }
      }
      __syncthreads();
      if (adding) {
        if (a0 == 0)
          for (uint32_t u = lane; u < K; u += 4) {
            const float w = stateS[(av * K + u) * kStateWords + 3].w;
            if (!(w > 0.0f)) continue;
            const float* t = recTrial + sj * recStride + 2u * (av * K + u);
            const float J = t[1];
            de = __fmaf_rn(w, t[0], de);
            if (!finiteS(J)) geomFinite = false;
            jmin = fminf(jmin, J);
          }
        for (uint32_t j = firstInc; j < kItemTets && a0 + j < sh.count[av]; j += 4) {
          const float* t = tetTrial + sj * tetStride + 3u * (av * kItemTets + j);
          const float J = t[2];
          de = __fmaf_rn(t[1], t[0], de);
          if (!finiteS(J)) geomFinite = false;
          jmin = fminf(jmin, J);
        }
      }
    }
    if (adding) {
      jmin = groupMin<4>(jmin, mask);
      const bool allFinite = __all_sync(mask, geomFinite);
      de = groupSum<4>(de, mask);
      if (lane == 0) {
        sh.jmin[sj][av] = jmin;
        sh.de[sj][av] = de;
        sh.finite[sj][av] = allFinite ? 1u : 0u;
      }
    }
    __syncthreads();
    if (evalCount > 0) {
      bt = firstBt;
      ta = firstTa;
      searching = true;
      for (uint32_t j = 0; j < evalCount && searching; ++j, ++bt) {
        if (!sh.finite[j][tid]) {
          status = kNonfinite;
          minTrialDet = 0.f;
          backtracks = bt;
          searching = false;
          break;
        }
        const float trialMin = fminf(controlMin, sh.jmin[j][tid]);
        minTrialDet = trialMin;
        if (trialMin > kDeterminantFloor) {
          const float3 tp = position + ta * dr.direction;
          const float3 td = tp - position;
          float energy = sh.de[j][tid];
          energy += inertia * (dot3(position - predV, td) + 0.5f * dot3(td, td)) + floorDelta(p, position.y, td.y);
          if (p.objectiveFlags != 0u) energy += objectiveDelta(p, b, v, position, td);
          evals += 1;
          const float tb = kArmijoC1 * dot3(grad, td);
          if (!finiteS(energy)) {
            status = kNonfinite;
            backtracks = bt;
            searching = false;
            break;
          }
          if (energy <= tb) {
            alpha = ta;
            acceptedDelta = energy;
            bound = tb;
            backtracks = bt;
            status = kAccepted;
            acceptedD = td;
            acceptedP = tp;
            searching = false;
            break;
          }
        }
        ta *= kBacktrackFactor;
      }
    }
    roundTrials = kTrials;
  }
  if (solving) {
    if (status == kLineSearchFailed) backtracks = kMaxBacktracks;
    tgt[v] = make_float4(acceptedP.x, acceptedP.y, acceptedP.z, 1.0f);
    b.finalUpdate[v] = scaledLength(acceptedD);
    float4* L = &b.local[4ull * v];
    const float4 l0 = make_float4(dr.direction.x, dr.direction.y, dr.direction.z, alpha);
    const float4 l1 = make_float4(dr.minEig * dr.scale, dr.scale, dr.shift * dr.scale, dr.shift);
    const float4 l2 = make_float4(acceptedDelta, bound, dr.gdd, dr.residual);
    const float4 l3 = make_float4(minTrialDet, float(backtracks), float(evals), float(status));
    L[0] = l0; L[1] = l1; L[2] = l2; L[3] = l3;
    localValid = finiteS(l0.x) && finiteS(l0.y) && finiteS(l0.z) && finiteS(l0.w) && finiteS(l1.x) &&
                 finiteS(l1.y) && finiteS(l1.z) && finiteS(l1.w) && finiteS(l2.x) && finiteS(l2.y) &&
                 finiteS(l2.z) && finiteS(l2.w) && finiteS(l3.x) && status != kNonfinite && l1.w >= 0.0f;
    shiftN = dr.shift;
    haveRecord = true;
  }
  // Local aggregates of reduceCandidate's vertex loop (jgs2-shader.ts:3689-3790),
  // per scene: folded in shared memory when the block's vertices share one
  // scene, otherwise added per vertex.
  const uint32_t blockScene = sh.scene[0];
  const bool oneScene = __syncthreads_and(tid >= n || !haveRecord || sh.scene[tid] == blockScene) != 0;
  if (haveRecord) {
    const bool failure = status == kShiftLimit || status == kNonDescent || status == kLineSearchFailed ||
                         status == kNonfinite || status == kCholeskyFailed;
    uint32_t trials = 0;
    if (status == kAccepted) trials = backtracks + 1;
    else if (status == kLineSearchFailed && backtracks == kMaxBacktracks) trials = kTrialCount;
    else if (status == kZeroGradient && backtracks > 0) trials = backtracks;
    else if (status == kNonfinite) trials = backtracks;  // a nonfinite trial never has J above the floor here
    const uint32_t skipped = trials - (trials < evals ? trials : evals);
    const uint32_t shiftBits = (shiftN > 0.0f && finiteS(shiftN)) ? __float_as_uint(shiftN) : 0u;
    FrameState* fs = &b.frames[sh.scene[tid]];
    uint32_t* fail = oneScene ? &sh.fail : &fs->localFailures;
    uint32_t* back = oneScene ? &sh.maxBack : &fs->localMaxBacktracks;
    uint32_t* skip = oneScene ? &sh.skip : &fs->localSkipped;
    uint32_t* ev = oneScene ? &sh.evals : &fs->localEvaluations;
    uint32_t* shift = oneScene ? &sh.maxShift : &fs->localMaxShift;
    uint32_t* valid = oneScene ? &sh.valid : &fs->localNumericsValid;
    if (failure) atomicAdd(fail, 1u);
    if (backtracks) atomicMax(back, backtracks);
    if (skipped) atomicAdd(skip, skipped);
    if (evals) atomicAdd(ev, evals);
    if (shiftBits) atomicMax(shift, shiftBits);
    if (!localValid) atomicAnd(valid, 0u);
  }
  __syncthreads();
  if (oneScene && tid == 0) {
    FrameState* fs = &b.frames[blockScene];
    if (sh.fail) atomicAdd(&fs->localFailures, sh.fail);
    if (sh.maxBack) atomicMax(&fs->localMaxBacktracks, sh.maxBack);
    if (sh.skip) atomicAdd(&fs->localSkipped, sh.skip);
    if (sh.evals) atomicAdd(&fs->localEvaluations, sh.evals);
    if (sh.maxShift) atomicMax(&fs->localMaxShift, sh.maxShift);
    if (!sh.valid) atomicAnd(&fs->localNumericsValid, 0u);
  }
}

// ---------------------------------------------------------------------------
// Graph-coloured sweep as one persistent kernel (jgs2-solver.ts:2275-2325,
// colour masks jgs2-shader.ts:3004-3012): for each colour, the vertex frames
// of the vertices the colour's solves read, a grid barrier, the in-place
// local solves of the colour's vertices, a grid barrier.  The grid is
// launched cooperatively (all blocks resident).  Each barrier is a bounded
// spin: a block that waits longer than `spinLimit` polls sets the sweep's
// error word and every block leaves at its next barrier, so the kernel always
// returns; the host reports JGS2_TIMEOUT at its next synchronisation.
struct SweepBarrier {
  uint32_t arrived, generation, error, pad;
};

// Bounded grid barrier; false when the sweep has failed (by this block's
// timeout or another's).
__device__ __forceinline__ bool gridBarrier(SweepBarrier* bar, uint32_t spinLimit) {
  __shared__ uint32_t sOk;
  __syncthreads();
  if (threadIdx.x == 0) {
    volatile SweepBarrier* vb = bar;
    const uint32_t gen = vb->generation;
    __threadfence();
    const uint32_t before = atomicAdd(&bar->arrived, 1u);
    if (before == gridDim.x - 1) {
      bar->arrived = 0u;
      __threadfence();
      atomicAdd(&bar->generation, 1u);
    } else {
      uint32_t spins = 0;
      while (vb->generation == gen && vb->error == 0u) {
        if (++spins > spinLimit) {
          atomicOr(&bar->error, 1u);
          break;
        }
        __nanosleep(32);
      }
    }
    __threadfence();
    sOk = vb->error == 0u ? 1u : 0u;
  }
  __syncthreads();
  return sOk != 0u;
}

template <int W, bool kExt>
__global__ void __launch_bounds__(kBlock, JGS2_SOLVE_MIN_BLOCKS)
    coloredSweepKernel(Buffers b, const DevParams* __restrict__ pp, float4* x, const uint32_t* __restrict__ colorVertices,
                       const uint32_t* __restrict__ colorOffsets, const uint32_t* __restrict__ needVertices,
                       const uint32_t* __restrict__ needOffsets, uint32_t colorCount, uint32_t V, uint32_t K,
                       uint32_t groupsPerBlock, int refreshAllFrames, SweepBarrier* bar, uint32_t spinLimit) {
  for (uint32_t c = 0; c < colorCount; ++c) {
    // Frames of the vertices this colour reads (every vertex after the
    // frame's last colour, so the stored frames match a full pass).
    const bool all = refreshAllFrames && c + 1 == colorCount;
    const uint32_t nb = needOffsets[c], ne = all ? nb + V : needOffsets[c + 1];
    for (uint32_t i = nb + blockIdx.x * blockDim.x + threadIdx.x; i < ne; i += gridDim.x * blockDim.x) {
      const uint32_t v = all ? i - nb : needVertices[i];
      const uint32_t scene = b.vertexScene[v];
      const DevParams& p = pp[scene];
      if (!p.active || latched(p, &b.frames[scene])) continue;
      storeFrame(b.vertexPack, v, vertexFrame<true>(b, x, v, p.rotationEpsilon), xyz(__ldca(x + v)));
    }
    if (!gridBarrier(bar, spinLimit)) return;
    const uint32_t cb = colorOffsets[c], count = colorOffsets[c + 1] - cb;
    const uint32_t chunks = (count + groupsPerBlock - 1) / groupsPerBlock;
    for (uint32_t chunk = blockIdx.x; chunk < chunks; chunk += gridDim.x)
      solveChunk<W, kExt, true>(b, pp, x, x, colorVertices + cb, count, K, 0, groupsPerBlock, chunk);
    if (!gridBarrier(bar, spinLimit)) return;
  }
}

// ---------------------------------------------------------------------------
// Grid-wide reductions.  The gate's blocks and the prologue's and the
// convergence pass's warps each fold their elements into one partial with a
// fixed tree; the last to take a ticket folds the scene's partials in a fixed
// order.  Results are deterministic for a given device; nothing waits.
struct GatePartial {
  double e0, e1;      // source / candidate assembled energy
  float minS, minC;   // minimum determinant, source / candidate
  uint32_t bits;      // AND of geometry / energy validity bits
  uint32_t pad;
};
constexpr uint32_t kGateBits = kSourceGeometryValid | kCandidateGeometryValid | kSourceEnergyValid |
                               kCandidateEnergyValid;

__device__ __forceinline__ GatePartial gateIdentity() { return {0.0, 0.0, kF32Max, kF32Max, kGateBits, 0u}; }
__device__ __forceinline__ void gateCombine(GatePartial& a, const GatePartial& b) {
  a.e0 += b.e0;
  a.e1 += b.e1;
  a.minS = fminf(a.minS, b.minS);
  a.minC = fminf(a.minC, b.minC);
  a.bits &= b.bits;
}

struct ConvPartial {
  double sq[6];     // squared norms: five components and their sum
  float scale[6];   // max-abs entries (validity of the robust norm)
  float maxUpdate;
  uint32_t valid;
};
__device__ __forceinline__ ConvPartial convIdentity() {
  ConvPartial p;
  for (int c = 0; c < 6; ++c) { p.sq[c] = 0.0; p.scale[c] = 0.0f; }
  p.maxUpdate = 0.0f;
  p.valid = 1u;
  return p;
}
__device__ __forceinline__ void convCombine(ConvPartial& a, const ConvPartial& b) {
  for (int c = 0; c < 6; ++c) {
    a.sq[c] += b.sq[c];
    a.scale[c] = fmaxf(a.scale[c], b.scale[c]);
  }
  a.maxUpdate = fmaxf(a.maxUpdate, b.maxUpdate);
  a.valid &= b.valid;
}

// One value from the other lane of a shuffle step, word by word.
template <class P>
__device__ __forceinline__ P shflDown(const P& v, unsigned offset) {
  static_assert(sizeof(P) % 4 == 0, "partials are moved as 32-bit words");
  uint32_t words[sizeof(P) / 4];
  memcpy(words, &v, sizeof(P));
#pragma unroll
  for (unsigned i = 0; i < sizeof(P) / 4; ++i) words[i] = __shfl_down_sync(0xffffffffu, words[i], offset);
  P r;
  memcpy(&r, words, sizeof(P));
  return r;
}

// Warp value in lane 0 (fixed tree).
template <class P, class C>
__device__ __forceinline__ P warpFold(P v, C combine) {
#pragma unroll
  for (unsigned o = 16; o > 0; o >>= 1) combine(v, shflDown(v, o));
  return v;
}

// Block value in thread 0 (fixed tree: lanes by shuffles, then the warps'
// values in one more shuffle tree).  `smem` holds one value per warp.  A tree
// in shared memory took a block barrier per level, seven at 128 threads, and
// blocks of small scenes do little else.
template <class P, class I, class C>
__device__ __forceinline__ P blockFold(P v, P* smem, I identity, C combine) {
  v = warpFold(v, combine);
  const unsigned warp = threadIdx.x / 32, lane = threadIdx.x & 31u;
  if (lane == 0) smem[warp] = v;
  __syncthreads();
  if (warp == 0) {
    v = lane < kBlock / 32 ? smem[lane] : identity();
#pragma unroll
    for (unsigned o = kBlock / 64; o > 0; o >>= 1) combine(v, shflDown(v, o));
  }
  __syncthreads();
  return v;
}

// Publishes the block partial at `slot`; returns true in every thread of the
// last of the `count` blocks sharing `ticket`.
template <class P>
__device__ __forceinline__ bool publishPartial(const P& blockValue, P* partials, uint32_t slot, uint32_t count,
                                               uint32_t* ticket, bool* isLast) {
  if (threadIdx.x == 0) {
    partials[slot] = blockValue;
    __threadfence();
    *isLast = atomicAdd(ticket, 1u) == count - 1;
  }
  __syncthreads();
  const bool last = *isLast;
  if (last) __threadfence();
  return last;
}

// Partials first, first + stride, ... below count, added in that order.
// Other blocks wrote them: they are read from L2, four of a thread's in
// flight at a time (one at a time, the 2 930 gate partials of six million
// tets kept the last block waiting for 23 L2 round trips).
template <class P, class C>
__device__ __forceinline__ void addPartials(P& acc, const P* partials, uint32_t first, uint32_t stride, uint32_t count,
                                            C combine) {
  static_assert(sizeof(P) % 16 == 0, "partials are read as 16-byte words");
  constexpr uint32_t kAhead = 4, kWords = sizeof(P) / 16;
  for (uint32_t k0 = first; k0 < count; k0 += stride * kAhead) {
    uint4 words[kAhead][kWords];
#pragma unroll
    for (uint32_t j = 0; j < kAhead; ++j) {
      const uint4* w = reinterpret_cast<const uint4*>(partials + min(k0 + stride * j, count - 1));
#pragma unroll
      for (uint32_t i = 0; i < kWords; ++i) words[j][i] = __ldcg(w + i);
    }
#pragma unroll
    for (uint32_t j = 0; j < kAhead; ++j) {
      P v;
      memcpy(&v, words[j], sizeof(P));
      if (k0 + stride * j < count) combine(acc, v);
    }
  }
}

// Folds partials[0, count) by a block (deterministic).
template <class P, class I, class C>
__device__ __forceinline__ P foldPartials(const P* partials, uint32_t count, P* smem, I identity, C combine) {
  P acc = identity();
  addPartials(acc, partials, threadIdx.x, blockDim.x, count, combine);
  return blockFold(acc, smem, identity, combine);
}

// Reduction over entries of one warp each (prologue and convergence): the
// last warp of 32 consecutive entries folds them into the group's partial and
// the last of those folds the scene's groups, so no warp reads more than a
// few partials per lane.  True, with the scene's value in lane 0 of `value`,
// on the scene's last warp; the tickets are then zero again.
template <class P, class I, class C>
__device__ __forceinline__ bool foldEntries(P& value, P* partials, P* groups, uint32_t* groupTickets,
                                            uint32_t* ticket, const RedBlock& rb, const SceneRange& sr, I identity,
                                            C combine) {
  const uint32_t lane = threadIdx.x & 31u;
  auto publish = [&](P* at, uint32_t* t, uint32_t count) {
    uint32_t last = 0;
    if (lane == 0) {
      *at = value;
      __threadfence();
      last = atomicAdd(t, 1u) == count - 1 ? 1u : 0u;
      if (last) *t = 0u;
    }
    last = __shfl_sync(0xffffffffu, last, 0);
    if (last) __threadfence();
    return last != 0u;
  };
  value = warpFold(value, combine);
  const uint32_t local = rb.slot - sr.convBase, group = local / 32, first = group * 32;
  const uint32_t inGroup = min(32u, sr.convBlocks - first), groupCount = (sr.convBlocks + 31) / 32;
  if (!publish(&partials[rb.slot], &groupTickets[sr.convGroupBase + group], inGroup)) return false;
  P acc = identity();
  addPartials(acc, partials + sr.convBase + first, lane, 32u, inGroup, combine);
  value = warpFold(acc, combine);
  if (groupCount == 1) return true;
  if (!publish(&groups[sr.convGroupBase + group], ticket, groupCount)) return false;
  acc = identity();
  addPartials(acc, groups + sr.convGroupBase, lane, 32u, groupCount, combine);
  value = warpFold(acc, combine);
  return true;
}

__device__ __forceinline__ void accumulateTet(GatePartial& acc, const TetRec& r, const M3& sF, const M3& cF) {
  const float sJ = mdet(sF), cJ = mdet(cF);
  const bool sgv = finiteS(sJ), cgv = finiteS(cJ);
  if (sgv) acc.minS = fminf(acc.minS, sJ); else acc.bits &= ~kSourceGeometryValid;
  if (cgv) acc.minC = fminf(acc.minC, cJ); else acc.bits &= ~kCandidateGeometryValid;
  bool sev = false, cev = false;
  if (sgv && sJ > kDeterminantFloor) {
    const float e = r.vol * snhEnergy(sF, r.lambda, r.mu);
    sev = finiteS(e);
    if (sev) acc.e0 += e;
  }
  if (cgv && cJ > kDeterminantFloor) {
    const float e = r.vol * snhEnergy(cF, r.lambda, r.mu);
    cev = finiteS(e);
    if (cev) acc.e1 += e;
  }
  if (!sev) acc.bits &= ~kSourceEnergyValid;
  if (!cev) acc.bits &= ~kCandidateEnergyValid;
}

// A cloth triangle as a gate element: its signed area stretch at the source
// and the candidate (candidateTetrahedron, jgs2-shader.ts:3507-3549), and its
// membrane energy, which the reference adds to the energy of the triangle's
// lowest vertex when that vertex's area stretch is above the floor and
// replaces the vertex energy by kF32Max otherwise (:2585-2621).
__device__ __forceinline__ void accumulateClothTri(GatePartial& acc, const ClothTri& t, const float4* __restrict__ s,
                                                   const float4* __restrict__ c, const ClothMaterial& m) {
  const float3 s0 = xyz(s[t.i0]), s1 = xyz(s[t.i1]), s2 = xyz(s[t.i2]);
  const float3 c0 = xyz(c[t.i0]), c1 = xyz(c[t.i1]), c2 = xyz(c[t.i2]);
  const float3 sn = clothRawNormal(s0, s1, s2), cn = clothRawNormal(c0, c1, c2);
  const float twice = 2.0f * t.area;
  const float ss = length3(sn) / twice;
  const float cm = length3(cn) / twice;
  const float cs = dot3(sn, cn) > 0.0f ? cm : -cm;
  const bool sgv = twice > 0.0f && finiteV(sn) && finiteS(ss);
  const bool cgv = twice > 0.0f && finiteV(cn) && finiteS(cs);
  if (sgv) acc.minS = fminf(acc.minS, ss); else acc.bits &= ~kSourceGeometryValid;
  if (cgv) acc.minC = fminf(acc.minC, cs); else acc.bits &= ~kCandidateGeometryValid;
  const float es = (twice > 0.0f && finiteS(ss) && ss > kDeterminantFloor) ? clothMembraneEnergy(t, s0, s1, s2, m)
                                                                            : kF32Max;
  const float ec = (twice > 0.0f && finiteS(cm) && cm > kDeterminantFloor) ? clothMembraneEnergy(t, c0, c1, c2, m)
                                                                            : kF32Max;
  if (finiteS(es)) acc.e0 += es; else acc.bits &= ~kSourceEnergyValid;
  if (finiteS(ec)) acc.e1 += ec; else acc.bits &= ~kCandidateEnergyValid;
}

// An active IPC candidate's barrier and friction energy at the source
// (source contact cache) and the candidate (target cache, or the source cache
// when the contact step collapsed to zero): ipcOwnedEnergy (:751-781), which
// the reference adds to the energy of the candidate's first unpinned vertex,
// and which becomes kF32Max for an invalid contact.
__device__ __forceinline__ void accumulateContact(GatePartial& acc, const Buffers& b, const DevParams& p,
                                                  float contactAlpha, uint32_t c, const float4* __restrict__ src,
                                                  const float4* __restrict__ tgt) {
  if (!b.contactFlag[c]) return;  // not in the active rows of this iteration
  const float near = b.contactNear[c], after = contactAlpha != 0.0f ? b.contactTargetNear[c] : near;
  if (ipcNearValid(near) && ipcNearValid(after) && !ipcNearFriction(near) &&
      !ipcBarrierActive(fabsf(near), p.ipcActivation) && !ipcBarrierActive(fabsf(after), p.ipcActivation))
    return;  // neither pose touches it: both energies are zero
  const float4* st = b.contactState + kContactStateWords * static_cast<size_t>(c);
  const ContactData ks = ipcCached(st[kContactSource], st[kContactSourceWeights]);
  const ContactData kc = contactAlpha != 0.0f ? ipcCached(st[kContactTarget], st[kContactTargetWeights]) : ks;
  const bool friction = p.ipcFriction > 0.0f && st[kContactLagged].w > 0.0f;
  auto energy = [&](const ContactData& k, const float4* __restrict__ x) {
    if (!k.valid) return kF32Max;
    if (!ipcBarrierActive(k.distance, p.ipcActivation) && !friction) return 0.0f;
    const float e = contactEnergy(b, p, c, k, x, 0xffffffffu, f3(0, 0, 0));
    return finiteS(e) ? e : kF32Max;
  };
  const float es = energy(ks, src), ec = energy(kc, tgt);
  if (finiteS(es)) acc.e0 += es; else acc.bits &= ~kSourceEnergyValid;
  if (finiteS(ec)) acc.e1 += ec; else acc.bits &= ~kCandidateEnergyValid;
}

// A hinge's bending energy at the source and the candidate (owned by its
// lowest vertex in the reference, :2623-2642).
__device__ __forceinline__ void accumulateHinge(GatePartial& acc, const float4* __restrict__ hinges, uint32_t h,
                                                const float4* __restrict__ s, const float4* __restrict__ c,
                                                float bending) {
  const uint4 q = hingeIndices(hinges, h);
  const float4 rest = __ldg(&hinges[2ull * h + 1]);
  const float es = clothBendingEnergy(xyz(s[q.x]), xyz(s[q.y]), xyz(s[q.z]), xyz(s[q.w]), rest, bending);
  const float ec = clothBendingEnergy(xyz(c[q.x]), xyz(c[q.y]), xyz(c[q.z]), xyz(c[q.w]), rest, bending);
  if (finiteS(es)) acc.e0 += es; else acc.bits &= ~kSourceEnergyValid;
  if (finiteS(ec)) acc.e1 += ec; else acc.bits &= ~kCandidateEnergyValid;
}

// Elements [x, y) of `n` that fall to a scene's reduction entry.
__device__ __forceinline__ uint2 blockShare(uint32_t n, const RedBlock& rb, const SceneRange& sr) {
  const uint64_t i = rb.slot - sr.convBase;
  return make_uint2(static_cast<uint32_t>(n * i / sr.convBlocks), static_cast<uint32_t>(n * (i + 1) / sr.convBlocks));
}

// ---------------------------------------------------------------------------
// Prologue: predict (jgs2-shader.ts:2660-2692), iteration-0 vertex frames and
// the source feasibility preflight (candidateTetrahedron + reduceCandidate on
// the accepted pose, jgs2-solver.ts:2240-2259).
//
// One warp per reduction entry: its vertices, and its share of the scene's
// tets, cloth triangles and hinges, so every warp has the same mix of work.
// kWide: a block per entry, whose eight warps first form the incident sums.
template <bool kWide>
__global__ void __launch_bounds__(kWide ? kWideBlock : kBlock) prologueKernel(Buffers b,
                                                                              const DevParams* __restrict__ pp) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t entry = kWide ? blockIdx.x : blockIdx.x * (kBlock / 32) + threadIdx.x / 32;
  if (entry >= b.convBlocks) return;  // uniform across the warp
  const RedBlock rb = b.convTable[entry];
  const SceneRange sr = b.scenes[rb.scene];
  const DevParams p = pp[rb.scene];
  if (!p.active) return;  // uniform across the scene's entries
  FrameState* fs = &b.frames[rb.scene];
  GatePartial acc = gateIdentity();
  IncidentShared* sh = nullptr;
  if constexpr (kWide) {
    __shared__ IncidentShared shared;
    sh = &shared;
    if (p.globalization) incidentBlockSums(b, p, b.pos[0], rb, sr, true, shared);
    if (threadIdx.x >= 32) return;
  }
  for (uint32_t k = rb.begin + lane; k < rb.end; k += 32) {
    const uint32_t i = sr.vOff + k;
    const float4 o = b.pos[0][i];
    b.old[i] = make_float4(o.x, o.y, o.z, 1.0f);
    const uint4 info = b.vinfo[i];
    const float4 rm = b.restMass[i];
    float3 pred = xyz(rm);
    if (!isPinned(info)) {
      const float3 vel = p.velocityDamping * xyz(b.velocity[i]);
      pred = xyz(o) + p.dt * vel + (p.dt * p.dt) * f3(p.gravity[0], p.gravity[1], p.gravity[2]);
    } else {
      b.velocity[i] = make_float4(0, 0, 0, 0);
    }
    const float4 target = make_float4(pred.x, pred.y, pred.z, distributedInertiaWeight(rm, info, p.invDt2));
    b.predicted[i] = target;
    b.vertexPack[4ull * i + 3] = target;
    b.finalUpdate[i] = 0.0f;
    // Co-rotated path: the iteration source is the inertial prediction; the
    // stable iteration source is the accepted pose.
    const float3 first = p.globalization ? xyz(o) : pred;
    b.pos[1][i] = make_float4(first.x, first.y, first.z, 1.0f);
    if (!p.globalization) continue;
    // Iteration-0 frames (and, for free vertices, the incident system).
    IncidentSums sums = incidentZero();
    if constexpr (kWide) sums = loadIncidentSums(sh->sums[k - rb.begin]);
    else incidentSums<true>(b, b.pos[0], info, sums);
    if (isPinned(info)) {
      const M3 favg = sums.total > 0.0f ? (1.0f / sums.total) * sums.avg : midentity();
      storeFrame(b.vertexPack, i, info.y == 0u ? midentity() : polarRotation(favg, p.rotationEpsilon), xyz(o));
    } else {
      storeFrameAndIncident(b, p, b.pos[0], i, info, sums, !kWide);
    }
    const float e = implicitEnergy(p, b, i, xyz(o), info);
    if (finiteS(e)) { acc.e0 += e; acc.e1 += e; }
    else acc.bits &= ~(kSourceEnergyValid | kCandidateEnergyValid);
  }
  if (p.globalization) {
    const uint2 tets = blockShare(sr.T, rb, sr);
    for (uint32_t k = tets.x + lane; k < tets.y; k += 32) {
      const TetRec r = loadTet(b.tets, sr.tOff + k);
      if (tetVerticesInBounds(r.idx, b.vertexTotal)) {
        const M3 F = deformationAt(r, b.pos[0]);
        accumulateTet(acc, r, F, F);
      }
    }
  }
  if (p.cloth) {
    const uint2 tris = blockShare(sr.C, rb, sr), hinges = blockShare(sr.H, rb, sr);
    for (uint32_t k = tris.x + lane; k < tris.y; k += 32)
      accumulateClothTri(acc, loadClothTri(b.clothTris, sr.cOff + k), b.pos[0], b.pos[0], clothMaterial(p));
    for (uint32_t k = hinges.x + lane; k < hinges.y; k += 32)
      accumulateHinge(acc, b.clothHinges, sr.hOff + k, b.pos[0], b.pos[0], p.clothBending);
  }
  if (!p.globalization) return;  // no preflight on the co-rotated path (uniform)
  GatePartial tot = acc;
  if (!foldEntries(tot, reinterpret_cast<GatePartial*>(b.gatePartials), reinterpret_cast<GatePartial*>(b.groupPartials),
                   b.groupTickets, &fs->prologueTicket, rb, sr, gateIdentity, gateCombine))
    return;
  if (lane != 0) return;
  uint32_t vb = tot.bits;
  if (sr.T == 0) vb &= ~(kSourceGeometryValid | kCandidateGeometryValid);
  const bool gv = (vb & kSourceGeometryValid) != 0u;
  const float e0 = float(tot.e0);
  const bool ev = (vb & kSourceEnergyValid) != 0u && finiteS(e0);
  const float m = tot.minS;
  const bool accepted = gv && m > kDeterminantFloor;
  uint32_t cbits = (vb & (kSourceGeometryValid | kCandidateGeometryValid)) | kLocalNumericsValid;
  if (gv) cbits |= kAcceptedMinimumValid;
  // predict clears the control records; the preflight then writes them with
  // history index 0 (jgs2-shader.ts:2687-2691, 3916-3953).
  fs->control[0] = make_float4(gv ? m : 0.f, gv ? m : 0.f, gv ? m : 0.f, float(cbits));
  fs->control[1] = make_float4(accepted ? 1.f : 0.f, accepted ? 0.f : 1.f, 0.f, 0.f);
  fs->control[2] = make_float4(ev ? e0 : 0.f, ev ? e0 : 0.f, ev ? e0 : 0.f, ev ? 1.f : 0.f);
  fs->control[3] = make_float4(0, 0, 0, 0);
}

// ---------------------------------------------------------------------------
// Gate: candidateTetrahedron (jgs2-shader.ts:3498-3601) + vertex energies
// (assembledVertexEnergy :3489-3496) + reduceCandidate (:3611-3955).
// kExt: some scene of the engine has cloth or contact candidates (their
// terms are compiled out otherwise).  JGS2_GATE_MIN_BLOCKS and
// JGS2_GATE_EXT_MIN_BLOCKS: blocks per SM each instantiation's register
// budget must allow.  For the tetrahedral gate, eight blocks (32 warps per SM
// for this gather-bound kernel) measured 22 % faster on the 100^3 cube than
// the compiler's choice (5 blocks), with bitwise the same results, and six
// and ten slower than eight; with the cloth and contact terms eight blocks
// cost the cloth drape 6 % of its gate time, so that instantiation keeps the
// five blocks the compiler chose for the kernel before the split.
#ifndef JGS2_GATE_MIN_BLOCKS
#define JGS2_GATE_MIN_BLOCKS 8
#endif
#ifndef JGS2_GATE_EXT_MIN_BLOCKS
#define JGS2_GATE_EXT_MIN_BLOCKS 5
#endif
template <bool kExt>
__global__ void __launch_bounds__(kBlock, kExt ? JGS2_GATE_EXT_MIN_BLOCKS : JGS2_GATE_MIN_BLOCKS)
    gateKernel(Buffers b, const DevParams* __restrict__ pp, const float4* __restrict__ src,
               const float4* __restrict__ tgt) {
  __shared__ GatePartial smem[kBlock / 32];
  __shared__ bool isLast;
  const RedBlock rb = b.gateTable[blockIdx.x];
  const SceneRange sr = b.scenes[rb.scene];
  const DevParams p = pp[rb.scene];
  FrameState* fs = &b.frames[rb.scene];
  if (!p.active || latched(p, fs)) return;  // uniform across the scene's blocks
  GatePartial acc = gateIdentity();
  // Contacts: element k takes candidates k, k + span, ... of the scene's
  // list (a single pass for static candidates, which the table covers).
  const uint32_t span = max(sr.gateSpan, 1u);
  const uint2 contacts =
      !kExt ? make_uint2(0u, 0u) : b.contactDynamic ? b.bpSpan[rb.scene] : make_uint2(sr.kOff, sr.KC);
  for (uint32_t k = rb.begin + threadIdx.x; k < rb.end; k += blockDim.x) {
    if (k < sr.T) {
      const TetRec r = loadTet(b.tets, sr.tOff + k);
      if (tetVerticesInBounds(r.idx, b.vertexTotal)) accumulateTet(acc, r, deformationAt(r, src), deformationAt(r, tgt));
    }
    if (k < sr.V) {
      const uint32_t i = sr.vOff + k;
      const uint4 info = b.vinfo[i];
      const float es = implicitEnergy(p, b, i, xyz(src[i]), info);
      const float ec = implicitEnergy(p, b, i, xyz(tgt[i]), info);
      if (finiteS(es)) acc.e0 += es; else acc.bits &= ~kSourceEnergyValid;
      if (finiteS(ec)) acc.e1 += ec; else acc.bits &= ~kCandidateEnergyValid;
    }
    if (kExt && p.cloth) {
      if (k < sr.C) accumulateClothTri(acc, loadClothTri(b.clothTris, sr.cOff + k), src, tgt, clothMaterial(p));
      if (k < sr.H) accumulateHinge(acc, b.clothHinges, sr.hOff + k, src, tgt, p.clothBending);
    }
    if (kExt && p.ipc)
      for (uint32_t c = k; c < contacts.y; c += span)
        accumulateContact(acc, b, p, fs->contactAlpha, contacts.x + c, src, tgt);
  }
  const GatePartial blk = blockFold(acc, smem, gateIdentity, gateCombine);
  GatePartial* partials = reinterpret_cast<GatePartial*>(b.gatePartials);
  if (!publishPartial(blk, partials, rb.slot, sr.gateBlocks, &fs->gateTicket, &isLast)) return;
  const GatePartial tot = foldPartials(partials + sr.gateBase, sr.gateBlocks, smem, gateIdentity, gateCombine);
  if (threadIdx.x != 0) return;
  uint32_t vb = tot.bits;
  if (__ldcg(&fs->localNumericsValid)) vb |= kLocalNumericsValid;
  const float eS = float(tot.e0), eC = float(tot.e1);
  if (!finiteS(eS)) vb &= ~kSourceEnergyValid;
  if (!finiteS(eC)) vb &= ~kCandidateEnergyValid;
  if (sr.T == 0) vb &= ~(kSourceGeometryValid | kCandidateGeometryValid);
  const float sm = tot.minS, cm = tot.minC;
  const bool sgv = (vb & kSourceGeometryValid) != 0u, cgv = (vb & kCandidateGeometryValid) != 0u;
  const bool sev = (vb & kSourceEnergyValid) != 0u, cev = (vb & kCandidateEnergyValid) != 0u;
  const bool accepted = (sgv && sm > kDeterminantFloor) && (cgv && cm > kDeterminantFloor);
  const float am = accepted ? cm : sm;
  const bool amv = accepted ? cgv : sgv;
  const float ae = accepted ? eC : eS;
  const bool aev = accepted ? cev : sev;
  if (amv) vb |= kAcceptedMinimumValid;
  uint32_t historyIndex = 0;
  const float packed = fs->control[1].w;
  if (finiteNonnegInt(packed, float(kHistoryCapacity))) historyIndex = static_cast<uint32_t>(packed);
  else vb &= ~kLocalNumericsValid;
  const uint32_t cb = vb & kValidityMask;
  const uint32_t failures = __ldcg(&fs->localFailures);
  fs->control[0] = make_float4(sgv ? sm : 0.f, cgv ? cm : 0.f, amv ? am : 0.f, float(cb));
  fs->control[1] = make_float4(accepted ? 1.f : 0.f, accepted ? 0.f : 1.f, float(failures), float(historyIndex));
  fs->control[2] = make_float4(sev ? eS : 0.f, cev ? eC : 0.f, aev ? ae : 0.f, (sev && cev) ? 1.f : 0.f);
  fs->control[3] = make_float4(__uint_as_float(__ldcg(&fs->localMaxShift)), float(__ldcg(&fs->localMaxBacktracks)),
                               float(__ldcg(&fs->localSkipped)), float(__ldcg(&fs->localEvaluations)));
  // Reset the sweep accumulators for the next iteration.
  fs->localFailures = 0u;
  fs->localMaxBacktracks = 0u;
  fs->localSkipped = 0u;
  fs->localEvaluations = 0u;
  fs->localMaxShift = 0u;
  fs->localNumericsValid = 1u;
  fs->gateTicket = 0u;
}

// ---------------------------------------------------------------------------
// applyCandidate (:3957-3983) + convergenceGradient (:3985-4097) +
// reduceConvergence (:4105-4486), and the next iteration's vertex frames.
// The five component norms are exact Euclidean norms accumulated in double;
// the reference forms the same norms in f32 as scale * sqrt(sum((g/scale)^2)).
// JGS2_CONV_MIN_BLOCKS: blocks per SM the convergence kernel's register
// budget must allow (the compiler's choice is 151 registers and 3 blocks).
// Four blocks (128 registers) measured 5 % faster on the 100^3 cube than the
// compiler's choice, with bitwise the same results; five and six were slower.
#ifndef JGS2_CONV_MIN_BLOCKS
#define JGS2_CONV_MIN_BLOCKS 4
#endif
// One warp per reduction entry.  kWide: a block per entry, whose eight warps
// first form the incident sums; then the first warp goes on alone.
template <bool kWide>
__global__ void __launch_bounds__(kWide ? kWideBlock : kBlock, kWide ? 2 : JGS2_CONV_MIN_BLOCKS)
    convergenceKernel(Buffers b, const DevParams* __restrict__ pp, const float4* __restrict__ src, float4* tgt,
                      int nextRotations) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t entry = kWide ? blockIdx.x : blockIdx.x * (kBlock / 32) + threadIdx.x / 32;
  if (entry >= b.convBlocks) return;  // uniform across the warp
  const RedBlock rb = b.convTable[entry];
  const SceneRange sr = b.scenes[rb.scene];
  const DevParams p = pp[rb.scene];
  FrameState* fs = &b.frames[rb.scene];
  if (!p.active || latched(p, fs)) return;  // uniform across the scene's entries
  const bool accepted = fs->control[1].x == 1.0f;
  const float4* __restrict__ acc = accepted ? tgt : src;
  const uint32_t V = sr.V;
  ConvPartial part = convIdentity();
  IncidentShared* sh = nullptr;
  if constexpr (kWide) {
    __shared__ IncidentShared shared;
    sh = &shared;
    incidentBlockSums(b, p, acc, rb, sr, nextRotations != 0, shared);
    if (threadIdx.x >= 32) return;
  }
  for (uint32_t k = rb.begin + lane; k < rb.end; k += 32) {
    const uint32_t v = sr.vOff + k;
    float upd = 0.0f;
    if (!accepted) {
      tgt[v] = src[v];
    } else {
      upd = scaledLength(xyz(tgt[v]) - xyz(src[v]));
    }
    b.finalUpdate[v] = upd;
    if (!(finiteS(upd) && upd >= 0.0f)) part.valid = 0u; else part.maxUpdate = fmaxf(part.maxUpdate, upd);
    const uint4 info = b.vinfo[v];
    IncidentSums sums = incidentZero();
    if (nextRotations || !isPinned(info)) {
      if constexpr (kWide) sums = loadIncidentSums(sh->sums[k - rb.begin]);
      else if (nextRotations) incidentSums<true>(b, acc, info, sums);
      else incidentSums<false>(b, acc, info, sums);
    }
    if (!isPinned(info)) {
      const float3 x = xyz(acc[v]);
      float3 comps[5];
      comps[0] = (b.restMass[v].w * p.invDt2) * (x - xyz(b.predicted[v]));
      Comp3& material = sums.grad;
      S3& hess = sums.hess;
      if (!kWide && p.cloth) {
        const uint4 cr = b.clothRange[v];
        if (nextRotations)
          clothLocalSystem<true>(b.clothTris, b.clothHinges, b.clothIncidence, cr, acc, clothMaterial(p), 0u, 1u,
                                 material, hess);
        else
          clothLocalSystem<false>(b.clothTris, b.clothHinges, b.clothIncidence, cr, acc, clothMaterial(p), 0u, 1u,
                                  material, hess);
      }
      comps[1] = cvalue(material);
      comps[2] = f3(0, 0, 0);
      comps[3] = f3(0, 0, 0);
      if (p.objectiveFlags != 0u) {
        if (p.objectiveFlags & 1u) comps[2] = -xyz(b.forces[v]);
        if (p.objectiveFlags & 2u) {
          const float4 t = b.targets[v];
          if (t.w > 0.0f) comps[3] = t.w * (x - xyz(t));
        }
      }
      comps[4] = f3(0, 0, 0);
      if (p.floorStiffness > 0.0f && x.y < p.floorHeight) comps[4].y = p.floorStiffness * (x.y - p.floorHeight);
      if (p.ipc) comps[4] = comps[4] + xyz(b.contactGrad[v]);  // contactGradientKernel
      float3 totalG = f3(0, 0, 0);
      bool tv = true;
#pragma unroll
      for (int c = 0; c < 5; ++c) {
        const bool ok = finiteV(comps[c]);
        const float3 val = ok ? comps[c] : f3(0, 0, 0);
        part.scale[c] = fmaxf(part.scale[c], fmaxf(fabsf(val.x), fmaxf(fabsf(val.y), fabsf(val.z))));
        part.sq[c] += double(val.x) * val.x + double(val.y) * val.y + double(val.z) * val.z;
        totalG = totalG + val;
        tv = tv && ok;
      }
      tv = tv && finiteV(totalG);
      if (tv) {
        part.scale[5] = fmaxf(part.scale[5], fmaxf(fabsf(totalG.x), fmaxf(fabsf(totalG.y), fabsf(totalG.z))));
        part.sq[5] += double(totalG.x) * totalG.x + double(totalG.y) * totalG.y + double(totalG.z) * totalG.z;
      } else {
        part.valid = 0u;
      }
      // The next iteration's frame and incident system from the same
      // deformation gradients (the accepted pose is the next source).
      if (nextRotations) storeIncident(b.incident, v, comps[1], hess);
    }
    if (nextRotations) {
      const M3 favg = sums.total > 0.0f ? (1.0f / sums.total) * sums.avg : midentity();
      storeFrame(b.vertexPack, v, info.y == 0u ? midentity() : polarRotation(favg, p.rotationEpsilon), xyz(acc[v]));
    }
  }
  ConvPartial tot = part;
  if (!foldEntries(tot, reinterpret_cast<ConvPartial*>(b.convPartials), reinterpret_cast<ConvPartial*>(b.groupPartials),
                   b.groupTickets, &fs->convTicket, rb, sr, convIdentity, convCombine))
    return;
  if (lane != 0) return;
  float norms[5];
  bool cnv = tot.valid != 0u;
  for (int c = 0; c < 5; ++c) {
    norms[c] = float(sqrt(tot.sq[c]));
    cnv = cnv && finiteS(norms[c]) && norms[c] >= 0.0f;
  }
  const float gnorm = float(sqrt(tot.sq[5]));
  const float den = fmaxf(1.0f, norms[0] + norms[1] + norms[2] + norms[3] + norms[4]);
  const float rel = gnorm / den;
  const bool rnv = cnv && finiteS(gnorm) && finiteS(den) && den >= 1.0f && finiteS(rel) && rel >= 0.0f;
  const float mu = tot.maxUpdate;
  const bool ssv = finiteS(p.sceneScale) && p.sceneScale >= 0.0f;
  const float nmu = mu / fmaxf(ssv ? p.sceneScale : 1.0e-12f, 1.0e-12f);
  const bool unv = tot.valid != 0u && ssv && finiteS(mu) && mu >= 0.0f && finiteS(nmu);
  const float4 geometry = fs->control[0];
  const uint32_t cb = controlBits(geometry.w) & kValidityMask;
  const bool sgv = (cb & kSourceGeometryValid) != 0u && finiteS(geometry.x);
  const bool cgv = (cb & kCandidateGeometryValid) != 0u && finiteS(geometry.y);
  const bool amv = (cb & kAcceptedMinimumValid) != 0u && finiteS(geometry.z);
  const bool lnv = (cb & kLocalNumericsValid) != 0u;
  const float4 accept = fs->control[1];
  const bool aav = finiteNonnegInt(accept.x, 1.0f), arv = finiteNonnegInt(accept.y, 1.0f);
  const bool lfv = finiteNonnegInt(accept.z, float(V));
  const bool hiv = finiteNonnegInt(accept.w, float(kHistoryCapacity));
  const bool aa = aav && accept.x == 1.0f, ar = arv && accept.y == 1.0f;
  const uint32_t failures = lfv ? static_cast<uint32_t>(accept.z) : 0u;
  const uint32_t hi = hiv ? static_cast<uint32_t>(accept.w) : 0u;
  const float4 cmx = fs->control[3];
  const bool cmv = finiteS(cmx.x) && cmx.x >= 0.0f && finiteNonnegInt(cmx.y, float(kMaxBacktracks)) &&
                   finiteNonnegInt(cmx.z, float(V) * float(kTrialCount)) &&
                   finiteNonnegInt(cmx.w, float(V) * float(kTrialCount));
  const bool fin = rnv && unv && sgv && cgv && amv && lnv && aav && arv && lfv && hiv && cmv;
  const bool rs = fin && rel <= p.residualTolerance;
  const bool us = fin && nmu <= p.normalizedUpdateTolerance;
  const bool conv = rs && us && aa && !ar && failures == 0u;
  if (hiv && hi < kHistoryCapacity) {
    float4* h = &fs->history[8 * hi];
    h[0] = fs->control[0];
    h[1] = make_float4(accept.x, accept.y, accept.z, ar ? 1.f : 0.f);
    h[2] = fs->control[2];
    h[3] = make_float4(cnv ? norms[0] : 0.f, cnv ? norms[1] : 0.f, cnv ? norms[2] : 0.f, cnv ? norms[3] : 0.f);
    h[4] = make_float4(cnv ? norms[4] : 0.f, rnv ? gnorm : 0.f, rnv ? den : 0.f, rnv ? rel : 0.f);
    h[5] = make_float4(unv ? mu : 0.f, unv ? nmu : 0.f, rs ? 1.f : 0.f, us ? 1.f : 0.f);
    h[6] = make_float4(conv ? 1.f : 0.f, fin ? 1.f : 0.f, float(hi), cmv ? cmx.x : 0.f);
    h[7] = make_float4(cmv ? cmx.y : 0.f, cmv ? cmx.z : 0.f, cmv ? cmx.w : 0.f, 1.f);
  }
  fs->control[1].w = float(hi + 1);
  if (conv && p.stopEnabled) fs->control[0].w = float(cb | kStopLatchBit);
}

// ---------------------------------------------------------------------------
// Epilogue: even-count copy (copyPosition, :4488-4496), optional body
// correction (:4498-4551), finalize (:4553-4589).
__global__ void __launch_bounds__(kBlock) bodyAccumulateKernel(Buffers b, const DevParams* __restrict__ pp,
                                                               const float4* __restrict__ finalPos, uint32_t V) {
  const uint32_t v = blockIdx.x * kBlock + threadIdx.x;
  if (v >= V || !pp[b.vertexScene[v]].active) return;
  float4 x = finalPos[v];
  if (finalPos != b.pos[0]) b.pos[0][v] = make_float4(x.x, x.y, x.z, 1.0f);
  const uint4 info = b.vinfo[v];
  const double m = fmax(double(b.restMass[v].w), 0.0);
  const float4 pr = b.predicted[v];
  // Per body: total mass, solved x/z moments, predicted x/z moments, pinned
  // count.  Double atomics: the summation order varies from run to run, so
  // the correction is reproducible to double rounding, not bitwise.
  double* acc = &b.bodyAccum[6ull * info.w];
  atomicAdd(&acc[0], m);
  atomicAdd(&acc[1], m * x.x);
  atomicAdd(&acc[2], m * x.z);
  atomicAdd(&acc[3], m * pr.x);
  atomicAdd(&acc[4], m * pr.z);
  if (isPinned(info)) atomicAdd(&acc[5], 1.0);
}

// accumulated: bodyAccumulateKernel ran (and left the final pose in pos[0]).
__global__ void __launch_bounds__(kBlock) finalizeKernel(Buffers b, const DevParams* __restrict__ pp,
                                                         const float4* __restrict__ finalPos, uint32_t V,
                                                         int accumulated) {
  const uint32_t v = blockIdx.x * kBlock + threadIdx.x;
  if (v >= V) return;
  const DevParams& p = pp[b.vertexScene[v]];
  if (!p.active) return;
  const uint4 info = b.vinfo[v];
  float4 x = accumulated ? b.pos[0][v] : finalPos[v];
  if (isPinned(info)) {
    if (!p.globalization) {
      const float4 rm = b.restMass[v];
      x = make_float4(rm.x, rm.y, rm.z, 1.0f);
    }
    b.pos[0][v] = make_float4(x.x, x.y, x.z, 1.0f);
    b.velocity[v] = make_float4(0, 0, 0, 0);
    return;
  }
  if (accumulated && p.bodyCorrection) {
    const double* acc = &b.bodyAccum[6ull * info.w];
    if (acc[5] == 0.0 && acc[0] > 0.0) {
      x.x += float((acc[3] - acc[1]) / acc[0]);
      x.z += float((acc[4] - acc[2]) / acc[0]);
    }
  }
  b.pos[0][v] = make_float4(x.x, x.y, x.z, 1.0f);
  const float3 o = xyz(b.old[v]);
  float3 vel = (xyz(x) - o) * p.invDt;
  if (p.floorStiffness > 0.0f && p.contactTangentialDamping > 0.0f && x.y <= p.floorHeight + p.contactMargin) {
    const float s = expf(-p.contactTangentialDamping * p.dt);
    vel.x *= s;
    vel.z *= s;
  }
  b.velocity[v] = make_float4(vel.x, vel.y, vel.z, 0.0f);
}

// ---------------------------------------------------------------------------
// Allocation-free variant of the gate.  Its reduction scratch is a static
// device array instead of solver buffers: a 256-byte header whose first word
// is the block ticket, then one GatePartial per block.  The ticket must be
// zero when a launch starts; module load zero-fills the array and the last
// block of every launch writes the ticket back to zero.  Two launches that
// overlap in time share the array and corrupt each other's result.
static_assert(sizeof(GatePartial) == kGatePartialBytes, "partial size");
static __device__ __align__(256) unsigned char gGateScratch[kGateScratchBytes];

// One element per thread (tet i and vertex i), so the grid, and with it the
// number of partials, grows with max(V, T); the launcher rejects sizes whose
// partials do not fit.  The sweep records are taken as cleared: no local
// failures, valid numerics, history slot 0, one skipped trial per vertex.
__global__ void __launch_bounds__(kBlock) gateScratchKernel(Buffers b, DevParams p, const float4* __restrict__ src,
                                                            const float4* __restrict__ tgt, uint32_t V, uint32_t T,
                                                            uint32_t C, uint32_t H, float4* __restrict__ control,
                                                            unsigned char* __restrict__ scratch) {
  __shared__ GatePartial smem[kBlock / 32];
  __shared__ bool isLast;
  uint32_t* ticket = reinterpret_cast<uint32_t*>(scratch);
  GatePartial* partials = reinterpret_cast<GatePartial*>(scratch + kGateScratchHeaderBytes);
  GatePartial acc = gateIdentity();
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < T) {
    const TetRec r = loadTet(b.tets, i);
    accumulateTet(acc, r, deformationAt(r, src), deformationAt(r, tgt));
  }
  if (i < V) {
    const uint4 info = b.vinfo[i];
    const float es = implicitEnergy(p, b, i, xyz(src[i]), info);
    const float ec = implicitEnergy(p, b, i, xyz(tgt[i]), info);
    if (finiteS(es)) acc.e0 += es; else acc.bits &= ~kSourceEnergyValid;
    if (finiteS(ec)) acc.e1 += ec; else acc.bits &= ~kCandidateEnergyValid;
  }
  if (i < C) accumulateClothTri(acc, loadClothTri(b.clothTris, i), src, tgt, clothMaterial(p));
  if (i < H) accumulateHinge(acc, b.clothHinges, i, src, tgt, p.clothBending);
  const GatePartial blk = blockFold(acc, smem, gateIdentity, gateCombine);
  if (!publishPartial(blk, partials, blockIdx.x, gridDim.x, ticket, &isLast)) return;
  const GatePartial tot = foldPartials(partials, gridDim.x, smem, gateIdentity, gateCombine);
  if (threadIdx.x != 0) return;
  uint32_t vb = tot.bits | kLocalNumericsValid;
  const float eS = float(tot.e0), eC = float(tot.e1);
  if (!finiteS(eS)) vb &= ~kSourceEnergyValid;
  if (!finiteS(eC)) vb &= ~kCandidateEnergyValid;
  if (T == 0) vb &= ~(kSourceGeometryValid | kCandidateGeometryValid);
  const float sm = tot.minS, cm = tot.minC;
  const bool sgv = (vb & kSourceGeometryValid) != 0u, cgv = (vb & kCandidateGeometryValid) != 0u;
  const bool sev = (vb & kSourceEnergyValid) != 0u, cev = (vb & kCandidateEnergyValid) != 0u;
  const bool accepted = (sgv && sm > kDeterminantFloor) && (cgv && cm > kDeterminantFloor);
  const float am = accepted ? cm : sm;
  const bool amv = accepted ? cgv : sgv;
  const float ae = accepted ? eC : eS;
  const bool aev = accepted ? cev : sev;
  if (amv) vb |= kAcceptedMinimumValid;
  const uint32_t cb = vb & kValidityMask;
  control[0] = make_float4(sgv ? sm : 0.f, cgv ? cm : 0.f, amv ? am : 0.f, float(cb));
  control[1] = make_float4(accepted ? 1.f : 0.f, accepted ? 0.f : 1.f, 0.f, 0.f);
  control[2] = make_float4(sev ? eS : 0.f, cev ? eC : 0.f, aev ? ae : 0.f, (sev && cev) ? 1.f : 0.f);
  control[3] = make_float4(0.f, 0.f, float(V), 0.f);
  *ticket = 0u;
}

}  // namespace

// ---------------------------------------------------------------------------
// Exact all-element oracle diagnostics (JGS2GpuOracleEvaluator,
// jgs2-diagnostics.ts:388-1146): per tet its frozen frame (the step's
// seven-step polar), energy, determinant and finiteness; per vertex the exact
// active-coordinate gradient, the diagonal block of the frozen global
// Hessian, the inertia, objective and floor energies and norms; one
// fixed-order reduction.  Opt-in; the frame loop never runs it.

__device__ __forceinline__ float finiteOr0(float v) { return finiteS(v) ? v : 0.0f; }
__device__ __forceinline__ float4 finite4(float3 v, float w) {
  return make_float4(finiteOr0(v.x), finiteOr0(v.y), finiteOr0(v.z), w);
}

// Co-rotated displacement of a tet's vertices in its frame R:
// R^T (x_l - centroid) - (X_l - rest centroid).
__device__ __forceinline__ void oracleDisplacement(const Buffers& b, const float4* __restrict__ x, const uint4& q,
                                                   const M3& R, float3 d[4], bool* finite) {
  float3 cur[4], rest[4];
  float3 cc = f3(0, 0, 0), rc = f3(0, 0, 0);
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    const uint32_t v = idxAt(q, l);
    cur[l] = xyz(x[v]);
    rest[l] = xyz(b.restMass[v]);
    cc = cc + 0.25f * cur[l];
    rc = rc + 0.25f * rest[l];
  }
  const M3 Rt = mtrans(R);
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    d[l] = mv(Rt, cur[l] - cc) - (rest[l] - rc);
    *finite = *finite && finiteV(cur[l]) && finiteV(rest[l]) && finiteV(d[l]);
  }
}

__global__ void __launch_bounds__(kBlock) oracleTetKernel(Buffers b, OracleParams q, const float4* __restrict__ x,
                                                          float4* __restrict__ rot, float4* __restrict__ metric) {
  const uint32_t k = blockIdx.x * kBlock + threadIdx.x;
  if (k >= q.T) return;
  const uint32_t t = q.tOff + k;
  const TetRec r = loadTet(b.tets, t);
  const M3 F = deformationAt(r, x);
  const float det = mdet(F);
  const M3 R = polarRotation(F, q.rotationEpsilon);
  bool finite = finiteM(F) && finiteS(det) && finiteM(R);
  float energy = 0.0f;
  if (q.corotated) {
    float3 d[4];
    oracleDisplacement(b, x, r.idx, R, d, &finite);
    const float* K = b.stiffness + 144ull * t;
#pragma unroll
    for (int row = 0; row < 4; ++row) {
      float3 lg = f3(0, 0, 0);
#pragma unroll
      for (int col = 0; col < 4; ++col) lg = lg + mv(stiffnessBlock(K, row, col), d[col]);
      finite = finite && finiteV(lg);
      energy += 0.5f * dot3(d[row], lg);
    }
  } else {
    energy = r.vol * snhEnergy(F, r.lambda, r.mu);
    const PiolaTerms pt = piolaTerms(F, r.lambda, r.mu);
    finite = finite && finiteM(piola(F, pt));
  }
  finite = finite && finiteS(energy);
  rot[3ull * k] = finite4(R.c0, 0.0f);
  rot[3ull * k + 1] = finite4(R.c1, 0.0f);
  rot[3ull * k + 2] = finite4(R.c2, 0.0f);
  metric[k] = make_float4(finiteOr0(energy), finiteOr0(det), finite ? 1.0f : 0.0f, 0.0f);
}

__global__ void __launch_bounds__(kBlock) oracleVertexKernel(Buffers b, OracleParams q, const float4* __restrict__ x,
                                                             const float4* __restrict__ rot,
                                                             float4* __restrict__ rec) {
  const uint32_t k = blockIdx.x * kBlock + threadIdx.x;
  if (k >= q.V) return;
  const uint32_t v = q.vOff + k;
  const uint4 info = b.vinfo[v];
  const float4 rm = b.restMass[v];
  const float3 cur = xyz(x[v]), pred = xyz(b.predicted[v]);
  const float3 diff = cur - pred;
  const float update = b.finalUpdate[v];
  const float floorDistance = cur.y - q.floorHeight;
  const bool active = !isPinned(info);
  float3 grad = f3(0, 0, 0), gIn = f3(0, 0, 0), gEl = f3(0, 0, 0), gExt = f3(0, 0, 0), gTgt = f3(0, 0, 0);
  float3 gFloor = f3(0, 0, 0);
  M3 H = mzero();
  float eIn = 0.0f, eExt = 0.0f, eTgt = 0.0f, eFloor = 0.0f, weight = 0.0f, mag = 0.0f;
  bool updateValid = false, floorActive = false;
  bool finite = finiteV(cur) && finiteV(pred) && finiteV(xyz(rm)) && finiteS(rm.w) && finiteS(update) &&
                finiteS(floorDistance);
  if (active) {
    weight = rm.w * q.invDt2;
    gIn = weight * diff;
    grad = gIn;
    H = weight * midentity();
    eIn = 0.5f * weight * dot3(diff, diff);
    mag = update;
    updateValid = update >= 0.0f;
    const float3 force = (q.objectiveFlags & 1u) ? xyz(b.forces[v]) : f3(0, 0, 0);
    gExt = -1.0f * force;
    eExt = -dot3(force, cur);
    grad = grad + gExt;
    const float4 target = (q.objectiveFlags & 2u) ? b.targets[v] : make_float4(0, 0, 0, 0);
    finite = finite && finiteV(force) && finiteS(target.w) && target.w >= 0.0f;
    if (target.w > 0.0f) {
      finite = finite && finiteV(xyz(target));
      const float3 res = cur - xyz(target);
      gTgt = target.w * res;
      eTgt = 0.5f * target.w * dot3(res, res);
      grad = grad + gTgt;
      H = H + target.w * midentity();
    }
    for (uint32_t a = 0; a < info.y; ++a) {
      const uint32_t entry = __ldg(&b.adjacency[info.x + a]);
      const uint32_t t = entry >> 2, slot = entry & 3u;
      const TetRec r = loadTet(b.tets, t);
      if (q.corotated) {
        const uint32_t kt = t - q.tOff;
        const M3 R = {xyz(rot[3ull * kt]), xyz(rot[3ull * kt + 1]), xyz(rot[3ull * kt + 2])};
        float3 d[4];
        oracleDisplacement(b, x, r.idx, R, d, &finite);
        const float* K = b.stiffness + 144ull * t;
        float3 lg = f3(0, 0, 0);
#pragma unroll
        for (int col = 0; col < 4; ++col) lg = lg + mv(stiffnessBlock(K, slot, col), d[col]);
        gEl = gEl + mv(R, lg);
        H = H + mm(mm(R, stiffnessBlock(K, slot, slot)), mtrans(R));
      } else {
        const M3 F = deformationAt(r, x);
        const PiolaTerms pt = piolaTerms(F, r.lambda, r.mu);
        const float3 g = shapeGradient(r, slot);
        gEl = gEl + r.vol * mv(piola(F, pt), g);
        S3 blk = szero();
        addIncidentBlock(blk, r, F, pt, g);
        H.c0 = H.c0 + f3(blk.xx, blk.xy, blk.xz);
        H.c1 = H.c1 + f3(blk.xy, blk.yy, blk.yz);
        H.c2 = H.c2 + f3(blk.xz, blk.yz, blk.zz);
      }
    }
    grad = grad + gEl;
    floorActive = q.floorStiffness > 0.0f && floorDistance < 0.0f;
    if (floorActive) {
      eFloor = 0.5f * q.floorStiffness * floorDistance * floorDistance;
      gFloor.y = q.floorStiffness * floorDistance;
      grad = grad + gFloor;
      H.c1.y += q.floorStiffness;
    }
  }
  const float gSq = dot3(grad, grad), inSq = dot3(gIn, gIn), elSq = dot3(gEl, gEl), flSq = dot3(gFloor, gFloor);
  finite = finite && finiteS(weight) && finiteS(eIn) && finiteS(eExt) && finiteS(eTgt) && finiteS(eFloor) &&
           finiteS(mag) && finiteV(grad) && finiteV(gIn) && finiteV(gEl) && finiteV(gExt) && finiteV(gTgt) &&
           finiteV(gFloor) && finiteM(H) && finiteS(gSq) && finiteS(inSq) && finiteS(elSq) &&
           finiteS(dot3(gExt, gExt)) && finiteS(dot3(gTgt, gTgt)) && finiteS(flSq);
  float4* o = rec + 9ull * k;
  o[0] = finite4(grad, active ? 1.0f : 0.0f);
  // Rows of the (symmetric) block with the energies beside them.
  o[1] = make_float4(finiteOr0(H.c0.x), finiteOr0(H.c1.x), finiteOr0(H.c2.x), finiteOr0(eIn));
  o[2] = make_float4(finiteOr0(H.c0.y), finiteOr0(H.c1.y), finiteOr0(H.c2.y), finiteOr0(eFloor));
  o[3] = make_float4(finiteOr0(H.c0.z), finiteOr0(H.c1.z), finiteOr0(H.c2.z), finiteOr0(mag));
  o[4] = make_float4(finiteOr0(gSq), finite ? 1.0f : 0.0f, finiteOr0(weight), updateValid ? 1.0f : 0.0f);
  o[5] = make_float4(finiteOr0(inSq), finiteOr0(elSq), finiteOr0(flSq), finiteOr0(floorDistance));
  o[6] = make_float4(floorActive ? 1.0f : 0.0f, 0.0f, 0.0f, 0.0f);
  o[7] = finite4(gExt, finiteOr0(eExt));
  o[8] = finite4(gTgt, finiteOr0(eTgt));
}

// reduceDiagnostics in one block: each thread folds a fixed stride of the
// records in double, then a fixed-order tree; deterministic.
__global__ void __launch_bounds__(1024) oracleReduceKernel(OracleParams q, const float4* __restrict__ metric,
                                                           const float4* __restrict__ rec, double* out) {
  __shared__ double sh[1024];
  double acc[kOracleSummaryWords];
#pragma unroll
  for (int i = 0; i < kOracleSummaryWords; ++i) acc[i] = 0.0;
  acc[11] = 0.0;                 // largest update
  acc[12] = 3.0e38;              // smallest determinant
  acc[13] = 3.0e38;              // smallest floor distance
  acc[16] = 1.0;                 // all active updates valid
  acc[17] = 1.0;                 // all finite
  for (uint32_t t = threadIdx.x; t < q.T; t += blockDim.x) {
    const float4 m = metric[t];
    acc[1] += m.x;
    acc[12] = fmin(acc[12], double(m.y));
    if (!(m.z >= 0.5f)) acc[17] = 0.0;
  }
  for (uint32_t v = threadIdx.x; v < q.V; v += blockDim.x) {
    const float4* o = rec + 9ull * v;
    const float4 g = o[0], r0 = o[1], r1 = o[2], r2 = o[3], m = o[4], c = o[5], fl = o[6], ext = o[7], tg = o[8];
    const bool active = g.w >= 0.5f;
    acc[0] += r0.w;
    acc[2] += ext.w;
    acc[3] += tg.w;
    acc[4] += r1.w;
    acc[5] += m.x;
    acc[6] += c.x;
    acc[7] += c.y;
    acc[8] += double(ext.x) * ext.x + double(ext.y) * ext.y + double(ext.z) * ext.z;
    acc[9] += double(tg.x) * tg.x + double(tg.y) * tg.y + double(tg.z) * tg.z;
    acc[10] += c.z;
    if (active) {
      acc[11] = fmax(acc[11], double(r2.w));
      acc[13] = fmin(acc[13], double(c.w));
      acc[15] += fl.x >= 0.5f ? 1.0 : 0.0;
      if (!(m.w >= 0.5f)) acc[16] = 0.0;
      acc[14] += 1.0;
    }
    if (!(m.y >= 0.5f)) acc[17] = 0.0;
  }
  for (int i = 0; i < kOracleSummaryWords; ++i) {
    sh[threadIdx.x] = acc[i];
    __syncthreads();
    for (uint32_t o = blockDim.x / 2; o > 0; o >>= 1) {
      if (threadIdx.x < o) {
        const double a = sh[threadIdx.x], c = sh[threadIdx.x + o];
        sh[threadIdx.x] = (i == 11) ? fmax(a, c) : (i == 12 || i == 13 || i == 16 || i == 17) ? fmin(a, c) : a + c;
      }
      __syncthreads();
    }
    if (threadIdx.x == 0) out[i] = sh[0];
    __syncthreads();
  }
}

inline uint32_t blocksFor(uint32_t n) { return (n + kBlock - 1) / kBlock; }

// SMs of the current device.
uint32_t smCount() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
  return static_cast<uint32_t>(sms);
}

// Eight lanes per vertex in the prologue and convergence passes, with the
// same bits.  Measured per convergence launch (events, about 6 us of which is
// the timing itself), eight lanes against one thread: 525 vertices 17 / 26 us,
// 2 688 vertices 19 / 27, 13 392 vertices 29 / 31, 27 360 vertices 41 / 35,
// 68 921 vertices 98 / 57: past about ten thousand vertices the threads hide
// each other's gathers.
//   With cloth the lanes pay longer, and it is the engine's whole size that
// decides, not its share of cloth: a cloth vertex has some 18 elements of
// several hundred operations, and by one thread even a few of them set the
// time of the launch (a 27 000-vertex solid alone 37 / 33 us, with a sheet of
// 81 vertices 40 / 51).  Sheets of 16 392 vertices 35 / 46, 22 809 46 / 50,
// 32 769 58 / 51; solids with sheets: 8 820 + 16 384 44 / 52, 19 683 + 10 201
// 49 / 52, 8 820 + 22 801 55 / 52.  A frame also has one prologue, where the
// lanes stop paying sooner (22 809-vertex sheet 64 / 56, 27 000 + 1 681 73 /
// 54): with four iterations a frame both forms take the same time between
// 28 000 and 31 000 vertices, whatever the mix.
constexpr uint32_t kWideVertices = 8192;
constexpr uint32_t kWideClothVertices = 28672;
bool wideIncident(const Buffers& b) { return b.vertexTotal <= (b.clothRange ? kWideClothVertices : kWideVertices); }

int launchPrologue(const Buffers& b, const DevParams* p, cudaStream_t s) {
  if (wideIncident(b)) prologueKernel<true><<<b.convBlocks, kWideBlock, 0, s>>>(b, p);
  else prologueKernel<false><<<(b.convBlocks + kBlock / 32 - 1) / (kBlock / 32), kBlock, 0, s>>>(b, p);
  return 1;
}

int launchTetPolar(const Buffers& b, const DevParams* p, const float4* src, uint32_t T, cudaStream_t s) {
  if (T == 0) return 0;
  tetPolarKernel<<<blocksFor(T), kBlock, 0, s>>>(b, p, src, T);
  return 1;
}

int launchCorotatedSolve(const Buffers& b, const DevParams* p, const float4* src, float4* tgt, const uint32_t* list,
                         uint32_t count, uint32_t K, cudaStream_t s) {
  if (count == 0) return 0;
  corotatedSolveKernel<<<(count + kCoVertices - 1) / kCoVertices, kBlock, 0, s>>>(b, p, src, tgt, list, count, K);
  return 1;
}

int launchVertexPolar(const Buffers& b, const DevParams* p, const float4* src, const uint32_t* list,
                      uint32_t count, cudaStream_t s) {
  if (count == 0) return 0;
  if (count <= kWideVertices)
    vertexPolarKernel<true><<<(count + kConvChunk - 1) / kConvChunk, kWideBlock, 0, s>>>(b, p, src, list, count);
  else vertexPolarKernel<false><<<blocksFor(count), kBlock, 0, s>>>(b, p, src, list, count);
  return 1;
}

// Lets `kernel` use `bytes` of dynamic shared memory on the current device.
// The limit is a property of the device's copy of the kernel, so it is set at
// every launch (once per captured frame): engines may be on several devices.
void allowShared(const void* kernel, uint32_t bytes) {
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
}

template <uint32_t kG, uint32_t kThreads, bool kJacobi, int kMin>
void launchItems(const Buffers& b, const DevParams* p, const float4* src, float4* tgt, const uint32_t* list,
                 uint32_t count, uint32_t K, uint32_t shift, cudaStream_t s) {
  static_assert(4 * kG <= kThreads, "four summing lanes per vertex");
  constexpr uint32_t trials = kG * kItemTets == kThreads ? kItemTrials : 1u;
  static_assert(4 * kG * trials <= kThreads, "four summing lanes per vertex and trial");
  const uint32_t limit = solveSharedBytes() - 12288;  // static shared memory of the kernel
  uint32_t groups = kG;
  while (groups > 1 && itemSharedBytes(groups, K, !kJacobi, trials) > limit) --groups;
  groups = std::max(1u, groups >> shift);
  allowShared(reinterpret_cast<const void*>(solveItemsKernel<kG, kThreads, kJacobi, kMin>), limit);
  solveItemsKernel<kG, kThreads, kJacobi, kMin>
      <<<(count + groups - 1) / groups, kThreads, itemSharedBytes(groups, K, !kJacobi, trials), s>>>(
          b, p, src, tgt, list, count, K, groups);
}

// The item form, or false where solveKernel's four lanes per vertex are the
// faster one.  Jacobi: eight vertices a block while one wave of two blocks per
// SM holds them, sixteen while that does (2 688 vertices: 27 us, 33 with
// eight, 37 with 32), then 32 on three blocks per SM.  Coloured lists: eight
// for three waves of blocks (3 650 vertices per colour: 60 us, 64 with sixteen,
// 71 with four lanes); past that four lanes (10 300 per colour: 90 us, 105 with
// sixteen, 117 with eight).  Those are six records a vertex; of other counts
// (1 to 66) the forms of eight and sixteen, and the coloured lists, are the
// faster ones throughout (525 vertices 24 records 21 / 46 us, 60 records
// 29 / 96; 2 750 vertices 12 records 23 / 34, 24 records 43 / 46), and the form
// of 32 where itemRoom says.
constexpr uint32_t kItemLargest = 40000;

// Whether an SM's shared memory holds as many blocks of 32 vertices by item (a
// record takes 296 bytes there, 240 with four lanes) as of four lanes, of which
// only three count, or one wave of blocks takes all vertices.  Measured per
// launch, items / four lanes: 27 000 vertices 6 records 63 / 75 us, 8 records
// 74 / 68, 9 records 85 / 90, 10 records 81 / 96, 12 records 152 / 112, 14
// records 157 / 134, 16 records 181 / 187, 24 records 251 / 264, 60 records
// 556 / 1 084; 39 304 vertices 8 records 119 / 101, 9 records 130 / 123, 10
// records 135 / 155, 12 records 244 / 172, 16 records 280 / 283.  At 8 and 9 records two blocks by item stand against three
// of four lanes, at 12 to 14 one against two; 8 820 vertices, which two blocks
// per SM take in one wave, 8 records 29 / 33, 9 records 31 / 41.
bool itemRoom(uint32_t count, uint32_t K) {
  constexpr uint32_t kG = 32;
  int dev = 0, perSm = 0;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&perSm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) != cudaSuccess) return true;
  auto resident = [&](size_t bytes) { return std::max<size_t>(1, perSm / (bytes + 1024)); };  // 1 KB is the system's
  const size_t items = resident(itemSharedBytes(kG, K, false, 1u) + sizeof(ItemShared<kG, 1u>));
  const size_t lanes = std::min<size_t>(3, resident(size_t(kG) * K * kSolveSlotBytes + 1024));
  return items >= lanes || count <= kG * items * smCount();
}
bool launchSolveItems(const Buffers& b, const DevParams* p, const float4* src, float4* tgt, const uint32_t* list,
                      uint32_t count, uint32_t K, bool jacobi, uint32_t shift, cudaStream_t s) {
  const uint32_t wave = 2 * smCount();  // blocks, two per SM
  if (jacobi) {
    if (count <= 8 * wave) launchItems<8, 192, true, 2>(b, p, src, tgt, list, count, K, shift, s);
    else if (count <= 16 * wave) launchItems<16, 192, true, 2>(b, p, src, tgt, list, count, K, shift, s);
    else if (count <= kItemLargest && itemRoom(count, K)) launchItems<32, 160, true, 3>(b, p, src, tgt, list, count, K, shift, s);
    else return false;
  } else {
    if (count <= 3 * 8 * wave) launchItems<8, 192, false, 2>(b, p, src, tgt, list, count, K, shift, s);
    else return false;
  }
  return true;
}

// solveKernel with its records cached in `shared` bytes.
template <int W, bool kExt>
void launchCached(const Buffers& b, const DevParams* p, const float4* src, float4* tgt, const uint32_t* list,
                  uint32_t count, uint32_t K, int ci, uint32_t groups, uint32_t blocks, uint32_t threads,
                  size_t shared, cudaStream_t s) {
  allowShared(reinterpret_cast<const void*>(solveKernel<W, kExt, true>), solveSharedBytes());
  solveKernel<W, kExt, true><<<blocks, threads, shared, s>>>(b, p, src, tgt, list, count, K, ci, groups);
}

int launchSolve(const Buffers& b, const DevParams* p, const float4* src, float4* tgt, const uint32_t* list,
                uint32_t count, uint32_t K, bool cachedIncident, cudaStream_t s) {
  if (count == 0) return 0;
  const bool cache = solveCachesRecords(K);
  const uint32_t fit = solveGroupsPerBlock(K);
  if (fit == 0) return 0;
  const uint32_t shift = std::min(b.solveShift, 2u);
  const uint32_t groups = std::max(1u, fit >> shift);
  const size_t smem = cache ? static_cast<size_t>(groups) * K * kSolveSlotBytes : 0;
  constexpr uint32_t perWarp = 32u / kGroup;
  const uint32_t threads = (groups + perWarp - 1) / perWarp * 32u;
  // One vertex per lane group: the line search makes per-vertex work uneven,
  // and the block scheduler balances it better than a fixed grid stride.
  const uint32_t blocks = std::max(1u, (count + groups - 1) / groups);
  // Contact-heavy engines (more than 64 candidate incidences of the static
  // superset per solved vertex on average, listed or not): a whole warp per
  // vertex over its active candidates.  A broad-phase engine decides on the
  // superset too, so it runs the variant its static twin runs.
  const uint64_t superset = b.contactDynamic ? b.bpSuperset : b.contactCount;
  const int ci = cachedIncident ? 1 : 0;
  if (b.contactIdx && superset * 4u > uint64_t(64) * count) {
    // Warps per block: an eighth of the vertices a 4-lane block of the same
    // cache budget would take (at most a full block).
    const uint32_t perVertex = static_cast<uint32_t>(K * kSolveSlotBytes);
    const uint32_t fit4 = std::min<uint32_t>(32u, (cache && perVertex) ? solveSharedBytes() / perVertex : 32u);
    const uint32_t wg = std::max(1u, std::min(std::max(1u, fit4 >> shift) * 4u / 32u, kBlock / 32u));
    const size_t wsmem = cache ? static_cast<size_t>(wg) * K * kSolveSlotBytes : 0;
    const uint32_t wb = std::max(1u, (count + wg - 1) / wg);
    if (cache)
      launchCached<32, true>(b, p, src, tgt, list, count, K, ci, wg, wb, wg * 32, wsmem, s);
    else
      solveKernel<32, true, false><<<wb, wg * 32, 0, s>>>(b, p, src, tgt, list, count, K, ci, wg);
  } else if (b.clothRange || b.contactIdx) {
    if (cache) launchCached<kGroup, true>(b, p, src, tgt, list, count, K, ci, groups, blocks, threads, smem, s);
    else solveKernel<kGroup, true, false><<<blocks, threads, 0, s>>>(b, p, src, tgt, list, count, K, ci, groups);
  } else if (cache && K > 0 && launchSolveItems(b, p, src, tgt, list, count, K, cachedIncident, shift, s)) {
  } else {
    if (cache) launchCached<kGroup, false>(b, p, src, tgt, list, count, K, ci, groups, blocks, threads, smem, s);
    else solveKernel<kGroup, false, false><<<blocks, threads, 0, s>>>(b, p, src, tgt, list, count, K, ci, groups);
  }
  return 1;
}

int launchColoredSweep(const Buffers& b, const DevParams* p, float4* x, const uint32_t* colorVertices,
                       const uint32_t* colorOffsets, const uint32_t* needVertices, const uint32_t* needOffsets,
                       uint32_t colorCount, uint32_t V, uint32_t K, uint32_t largestColor, uint32_t largestNeed,
                       bool refreshAllFrames, void* barrier, uint32_t spinLimit, cudaStream_t s) {
  const uint32_t fit = solveGroupsPerBlock(K);
  if (fit == 0 || colorCount == 0) return 0;
  if (!solveCachesRecords(K)) return -1;  // the sweep kernel caches records
  const uint32_t groups = std::max(1u, fit >> std::min(b.solveShift, 2u));
  const size_t smem = static_cast<size_t>(groups) * K * kSolveSlotBytes;
  constexpr uint32_t perWarp = 32u / kGroup;
  const uint32_t threads = (groups + perWarp - 1) / perWarp * 32u;
  const bool ext = b.clothRange || b.contactIdx;
  const void* fn = ext ? reinterpret_cast<const void*>(coloredSweepKernel<kGroup, true>)
                       : reinterpret_cast<const void*>(coloredSweepKernel<kGroup, false>);
  allowShared(fn, solveSharedBytes());
  int device = 0, sms = 0, perSm = 0;
  cudaGetDevice(&device);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, fn, static_cast<int>(threads), smem) != cudaSuccess ||
      perSm <= 0 || sms <= 0)
    return -1;
  // As many blocks as the widest phase can use: every colour's solves in one
  // wave of chunks (else the launch-per-colour encoding is the better one),
  // the frames spread at one vertex per thread.
  const uint32_t capacity = static_cast<uint32_t>(perSm * sms);
  const uint32_t chunks = (largestColor + groups - 1) / groups;
  if (chunks > capacity) return -1;
  const uint32_t frameBlocks = (std::max(largestNeed, refreshAllFrames ? V : 0u) + threads - 1) / threads;
  const uint32_t grid = std::max(1u, std::min(capacity, std::max(chunks, frameBlocks)));
  // A cooperative grid: every block resident, so the barriers can complete.
  cudaMemsetAsync(barrier, 0, sizeof(SweepBarrier), s);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  SweepBarrier* bar = static_cast<SweepBarrier*>(barrier);
  const int all = refreshAllFrames ? 1 : 0;
  cudaError_t e;
  if (ext)
    e = cudaLaunchKernelEx(&cfg, coloredSweepKernel<kGroup, true>, b, p, x, colorVertices, colorOffsets, needVertices,
                           needOffsets, colorCount, V, K, groups, all, bar, spinLimit);
  else
    e = cudaLaunchKernelEx(&cfg, coloredSweepKernel<kGroup, false>, b, p, x, colorVertices, colorOffsets,
                           needVertices, needOffsets, colorCount, V, K, groups, all, bar, spinLimit);
  return e == cudaSuccess ? 2 : -1;
}

size_t sweepBarrierBytes() { return sizeof(SweepBarrier); }

bool boundsChecked() { return JGS2_BOUNDS_CHECKS != 0; }

cudaError_t takeBoundsViolation(uint32_t* site) {
  *site = 0;
#if JGS2_BOUNDS_CHECKS
  cudaError_t e = cudaMemcpyFromSymbol(site, gBoundsViolation, sizeof(uint32_t));
  if (e != cudaSuccess || *site == 0) return e;
  const uint32_t zero = 0;
  return cudaMemcpyToSymbol(gBoundsViolation, &zero, sizeof(uint32_t));
#else
  return cudaSuccess;
#endif
}

uint32_t solveSharedBytes() {
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) optin = 48 * 1024;
  return static_cast<uint32_t>(optin - 1024);  // static shared memory of the kernel
}

bool solveCachesRecords(uint32_t K) { return static_cast<size_t>(K) * kSolveSlotBytes <= kSolveCacheBytesPerVertex; }

uint32_t solveGroupsPerBlock(uint32_t K) {
  // Shared memory holds one cached record state per cubature record of each
  // vertex in the block; wide records are recomputed instead of cached.
  uint32_t groups = (kBlock / 32) * (32 / kGroup);
  if (!solveCachesRecords(K)) return groups;
  const uint32_t perVertex = static_cast<uint32_t>(K * kSolveSlotBytes);
  if (perVertex > 0) groups = std::min<uint32_t>(groups, solveSharedBytes() / perVertex);
  return groups;
}

int launchContactLag(const Buffers& b, const DevParams* p, cudaStream_t s) {
  if (b.contactCount == 0) return 0;
  contactLagKernel<<<blocksFor(b.contactCount), kBlock, 0, s>>>(b, p);
  return 1;
}

int launchContactRows(const Buffers& b, const DevParams* p, const float4* src, uint32_t V, cudaStream_t s) {
  if (b.contactCount == 0) return 0;
  contactFlagKernel<<<blocksFor(b.contactCount), kBlock, 0, s>>>(b, p, src);
  contactRowsKernel<<<(V + kBlock / 32 - 1) / (kBlock / 32), kBlock, 0, s>>>(b, p, V);
  return 2;
}

int launchContactGradient(const Buffers& b, const DevParams* p, const float4* src, const float4* tgt, uint32_t V,
                          cudaStream_t s) {
  if (b.contactCount == 0) return 0;
  contactGradientKernel<<<(V + kBlock / 32 - 1) / (kBlock / 32), kBlock, 0, s>>>(b, p, src, tgt, V);
  return 1;
}

// Candidate kernels: one thread per static candidate, or a grid that strides
// over the broad phase's list (its count is on the device).
uint32_t candidateBlocks(const Buffers& b) {
  const uint32_t n = blocksFor(b.contactCount);
  return b.contactDynamic ? std::min(n, smCount() * 16u) : n;
}

int launchContactStep(const Buffers& b, const DevParams* p, const float4* src, const float4* tgt, cudaStream_t s) {
  if (b.contactCount == 0) return 0;
  // Lists of many candidates a vertex: the lengths once per vertex first.
  if (b.contactDynamic) {
    contactMoveKernel<<<blocksFor(b.vertexTotal), kBlock, 0, s>>>(b, src, tgt, b.vertexTotal);
    contactStepKernel<true><<<candidateBlocks(b), kBlock, 0, s>>>(b, p, src, tgt);
    return 2;
  }
  contactStepKernel<false><<<candidateBlocks(b), kBlock, 0, s>>>(b, p, src, tgt);
  return 1;
}

int launchContactApply(const Buffers& b, const DevParams* p, const float4* src, float4* tgt, uint32_t V,
                       bool validated, cudaStream_t s) {
  if (b.contactCount == 0) return 0;
  contactApplyKernel<<<blocksFor(V), kBlock, 0, s>>>(b, p, src, tgt, V, validated ? 1 : 0);
  return 1;
}

int launchContactValidate(const Buffers& b, const DevParams* p, const float4* tgt, cudaStream_t s) {
  if (b.contactCount == 0) return 0;
  contactValidateKernel<<<candidateBlocks(b), kBlock, 0, s>>>(b, p, tgt);
  return 1;
}

int launchContactFeatures(const float* points, const uint32_t* types, uint32_t n, float* out, uint32_t* wide,
                          cudaStream_t s) {
  if (n == 0) return 0;
  contactFeatureKernel<<<(n + kBlock - 1) / kBlock, kBlock, 0, s>>>(points, types, n, out, wide);
  return 1;
}

int launchContactPromote(const Buffers& b, const DevParams* p, cudaStream_t s) {
  if (b.contactCount == 0) return 0;
  contactPromoteKernel<<<candidateBlocks(b), kBlock, 0, s>>>(b, p);
  return 1;
}

uint32_t broadPhaseSortPasses(uint32_t V) {
  uint32_t bits = 1;
  while (bits < 32 && (V >> bits) != 0u) ++bits;  // keys 0..V, the sentinel V included
  return (bits + 7) / 8;
}

int launchBroadPhase(const Buffers& b, const DevParams* p, const float4* src, uint32_t V, bool first,
                     cudaStream_t s) {
  if (!b.contactDynamic || b.contactCount == 0) return 0;
  const uint32_t triBlocks = blocksFor(b.bpTriTotal), edgeBlocks = blocksFor(b.bpEdgeTotal);
  bpBoxesKernel<<<triBlocks + edgeBlocks + blocksFor(V), kBlock, 0, s>>>(b, p, src, triBlocks, edgeBlocks, V);
  const uint32_t triSupers = (b.bpTriTotal + kBpChunk * kBpChunk - 1) / (kBpChunk * kBpChunk);
  const uint32_t edgeSupers = (b.bpEdgeTotal + kBpChunk * kBpChunk - 1) / (kBpChunk * kBpChunk);
  bpSuperKernel<<<(triSupers + edgeSupers + kBlock / 32 - 1) / (kBlock / 32), kBlock, 0, s>>>(b, triSupers,
                                                                                              edgeSupers);
  const uint32_t rowBlocks = (b.bpRowTotal + kBlock / 32 - 1) / (kBlock / 32);
  const int f = first ? 1 : 0;
  bpRowsKernel<false><<<rowBlocks, kBlock, 0, s>>>(b, p, src, f);
  bpScanKernel<<<1, kScanThreads, 0, s>>>(b, p, f);
  bpRowsKernel<true><<<rowBlocks, kBlock, 0, s>>>(b, p, src, f);
  bpInitKernel<<<candidateBlocks(b), kBlock, 0, s>>>(b, p, src, f);
  const uint32_t tiles = static_cast<uint32_t>((4ull * b.contactCount + kSortTile - 1) / kSortTile);
  for (uint32_t pass = 0; pass < b.bpSortPasses; ++pass) {
    const uint32_t in = pass & 1u, out = in ^ 1u;
    bpSortHistKernel<<<tiles, kSortThreads, 0, s>>>(b.bpKeys[in], b.bpStatus, 8u * pass, b.bpHist);
    bpSortScanKernel<<<256, kScanThreads, 0, s>>>(b.bpStatus, b.bpHist);
    const auto scatter = pass == 0 ? bpSortScatterKernel<true> : bpSortScatterKernel<false>;
    scatter<<<tiles, kSortThreads, 0, s>>>(b.bpKeys[in], b.bpVals[in], b.bpKeys[out], b.bpVals[out], b.bpStatus,
                                           8u * pass, b.bpHist);
  }
  const uint32_t segBlocks = std::min(blocksFor(b.contactCount), smCount() * 16u);
  bpSegmentsKernel<<<segBlocks, kBlock, 0, s>>>(b, b.bpKeys[b.bpSortPasses & 1u]);
  return 7 + 3 * static_cast<int>(b.bpSortPasses);
}

int launchOracleDiagnostics(const Buffers& b, const OracleParams& q, float4* tetRot, float4* tetMetric,
                            float4* vertexRecords, double* summary, cudaStream_t s) {
  int n = 0;
  if (q.T) {
    oracleTetKernel<<<blocksFor(q.T), kBlock, 0, s>>>(b, q, b.pos[0], tetRot, tetMetric);
    ++n;
  }
  if (q.V) {
    oracleVertexKernel<<<blocksFor(q.V), kBlock, 0, s>>>(b, q, b.pos[0], tetRot, vertexRecords);
    ++n;
  }
  oracleReduceKernel<<<1, 1024, 0, s>>>(q, tetMetric, vertexRecords, summary);
  return n + 1;
}

int launchCopy(const Buffers& b, const DevParams* p, const float4* src, float4* dst, uint32_t V, cudaStream_t s) {
  copyKernel<<<blocksFor(V), kBlock, 0, s>>>(b, p, src, dst, V);
  return 1;
}

int launchGate(const Buffers& b, const DevParams* p, const float4* src, const float4* tgt, cudaStream_t s) {
  if (b.clothRange || b.contactIdx)
    gateKernel<true><<<b.gateBlocks, kBlock, 0, s>>>(b, p, src, tgt);
  else
    gateKernel<false><<<b.gateBlocks, kBlock, 0, s>>>(b, p, src, tgt);
  return 1;
}

int launchConvergence(const Buffers& b, const DevParams* p, const float4* src, float4* tgt,
                      bool computeNextRotations, cudaStream_t s) {
  const int next = computeNextRotations ? 1 : 0;
  if (wideIncident(b)) convergenceKernel<true><<<b.convBlocks, kWideBlock, 0, s>>>(b, p, src, tgt, next);
  else
    convergenceKernel<false><<<(b.convBlocks + kBlock / 32 - 1) / (kBlock / 32), kBlock, 0, s>>>(b, p, src, tgt, next);
  return 1;
}

int launchEpilogue(const Buffers& b, const DevParams* p, const float4* finalPos, uint32_t V, bool bodyCorrection,
                   uint32_t bodies, cudaStream_t s) {
  int n = 0;
  if (bodyCorrection) {
    cudaMemsetAsync(b.bodyAccum, 0, sizeof(double) * 6ull * bodies, s);
    bodyAccumulateKernel<<<blocksFor(V), kBlock, 0, s>>>(b, p, finalPos, V);
    ++n;
  }
  finalizeKernel<<<blocksFor(V), kBlock, 0, s>>>(b, p, finalPos, V, bodyCorrection ? 1 : 0);
  return n + 1;
}

cudaError_t gateScratchAddress(void** out) { return cudaGetSymbolAddress(out, gGateScratch); }

uint32_t gateScratchMaxElements() { return kGateScratchMaxBlocks * static_cast<uint32_t>(kBlock); }

int launchGateScratch(const Buffers& b, const DevParams& p, const float4* predicted, const float4* src,
                      const float4* tgt, uint32_t V, uint32_t T, uint32_t C, uint32_t H, float4* control,
                      void* scratch, cudaStream_t s) {
  const uint32_t n = std::max(std::max(T, V), std::max(C, H));
  if (n == 0 || n > gateScratchMaxElements()) return 0;
  Buffers view = b;
  view.predicted = const_cast<float4*>(predicted);
  gateScratchKernel<<<blocksFor(n), kBlock, 0, s>>>(view, p, src, tgt, V, T, C, H, control,
                                                   static_cast<unsigned char*>(scratch));
  return 1;
}

}  // namespace jgs2
