// Batched hit iteration (vklIterateHitsN) of float and coded attributes with
// the trilinear filter (any other attribute or filter: k_iterate.cu).
//
// hitNextWith (iterate.cuh) runs each ray's loop nest (DDA, march, NaN
// nudges, bisection) to completion, so the 32 rays of a warp are soon in
// different loops.  Here a warp's lanes share one loop whose round is
//   1. the sample that arrived is tested; a lane whose step crosses no
//      isovalue moves on at once, any other goes through a state machine
//      with exactly intersectBisection's steps;
//   2. a lane that needs its next interval takes one DDA step: lanes in
//      empty space do not hold up lanes that march (run to its next
//      interval, every round waited for the lane with the longest way
//      through empty space; one step a round measured 8.75 ms, two 9.3,
//      six 11.2, and holding samples back until 8 or 24 lanes want one 8.9
//      and 9.5);
//   3. every lane that needs a sample takes it at one call site.
// Each lane performs exactly the steps, samples and comparisons of
// hitNextWith in the same order, so hits are identical.  The kernels are
// persistent: a warp owns every numWarps-th block of 32 rays, and a lane that
// completes a ray takes the next one its warp has left, so neither a lane
// nor a warp idles behind the longest ray (12.0 -> 9.3 ms).
// 400,003 random rays through the 1024^3 shells, two isovalues: 27.3 -> 8.75
// ms.  Bound by instruction issue of diverging lanes (6 of 32 active).
#include <algorithm>
#include <type_traits>

#include "iterate.cuh"
#include "kernels.h"
#include "objects.h"

namespace vklcuda {

namespace {

constexpr int kBlock     = 128;
constexpr int kHitValues = 32;  // isovalues kept in shared memory
// 4 x 128 threads per SM: 128 registers, without spills for float leaves and
// with 24 to 72 bytes of them for coded ones (400,003 random rays, 1024^3
// shells, float: 8.75 ms; three: 10.3; five, spilling: 15.1 ms before the
// warp's ray pool).
constexpr int kHitMinBlocks = 4;

__device__ __forceinline__ f3 ld3(const float *p, uint64_t i)
{
  return {__ldg(p + 3 * i), __ldg(p + 3 * i + 1), __ldg(p + 3 * i + 2)};
}

enum WalkResult { kWalkEnd, kWalkEmpty, kWalkInterval };

// One step at a time of intervalNext over a sparse volume at full depth
// (elementary cells in leaves).  The DDA state of all four levels stays in
// registers; the level-2 node of the last query and its last leaf are kept,
// so a step within a leaf queries nothing and one within a 128^3 node loads
// one voxel and its range instead of three dependent ones.
struct SparseWalk {
  static constexpr int L = (int)kNumLevels - 1;
  f3 org, dir;
  DdaCell<L> d;
  float tMax;
  uint32_t budget;
  uint32_t nodeKey[3], node;  // node ~0: none
  uint32_t leafKey[3];
  uint32_t leaf;  // 0: none

  __device__ __forceinline__ void query(const DevGrid &g, uint32_t attr, const DevValueRanges &vr, uint32_t &level,
                                        bool &empty)
  {
    const uint32_t x = d.id[L][0], y = d.id[L][1], z = d.id[L][2];
    if (leaf && (((x ^ leafKey[0]) | (y ^ leafKey[1]) | (z ^ leafKey[2])) >> 3) == 0) {
      level = kNumLevels - 1;
      empty = false;
      return;
    }
    if (node == ~0u || (((x ^ nodeKey[0]) | (y ^ nodeKey[1]) | (z ^ nodeKey[2])) >> 7) != 0) {
      node       = ~0u;
      uint32_t n = 0;
#pragma unroll
      for (uint32_t l = 0; l < 2; ++l) {
        const uint32_t vo = (uint32_t)(offsetToLinear(l, x, y, z) + n * levelNumVoxels(l));
        const uint64_t v  = __ldg(g.levels[l].voxels + vo);
        const float2 r =
            __ldg((const float2 *)g.levels[l].valueRange + ((uint64_t)vo * g.numAttributes + attr));
        level = l;
        empty = voxelIsEmpty(v) || !rangesOverlap(vr, r.x, r.y);
        if (empty)
          return;
        if (voxelIsLeaf(v)) {
          level = l + 1;
          return;
        }
        n = (uint32_t)voxelChildIndex(v);
      }
      node       = n;
      nodeKey[0] = x;
      nodeKey[1] = y;
      nodeKey[2] = z;
    }
    const uint32_t vo = (uint32_t)(offsetToLinear(2, x, y, z) + node * levelNumVoxels(2));
    const uint64_t v  = __ldg(g.levels[2].voxels + vo);
    const float2 r    = __ldg((const float2 *)g.levels[2].valueRange + ((uint64_t)vo * g.numAttributes + attr));
    level             = 2;
    empty             = voxelIsEmpty(v) || !rangesOverlap(vr, r.x, r.y);
    if (!empty && voxelIsLeaf(v)) {
      level      = kNumLevels - 1;
      leaf       = 1;
      leafKey[0] = x;
      leafKey[1] = y;
      leafKey[2] = z;
    }
  }

  // hddaStep from `level`
  __device__ __forceinline__ void step(uint32_t level)
  {
    uint32_t b[3] = {0, 0, 0};
#pragma unroll
    for (int l = 0; l <= L; ++l)
      if (level == (uint32_t)l) {
#pragma unroll
        for (int a = 0; a < 3; ++a)
          b[a] = d.id[l][a];
        ddaStepCell(d, l);
#pragma unroll
        for (int a = 0; a < 3; ++a)
          b[a] = d.id[l][a] - b[a];
      }
    if (level < (uint32_t)L) {  // ddaReinitBelow
      const float d3[3] = {dir.x, dir.y, dir.z};
      const float g3[3] = {org.x, org.y, org.z};
      float oo[3]       = {org.x + d.t * dir.x, org.y + d.t * dir.y, org.z + d.t * dir.z};
      if (b[0] != 0)
        oo[0] = oo[0] + (float)dirSign(d3[0]) * 1e-2f;
      else if (b[1] != 0)
        oo[1] = oo[1] + (float)dirSign(d3[1]) * 1e-2f;
      else
        oo[2] = oo[2] + (float)dirSign(d3[2]) * 1e-2f;
#pragma unroll
      for (int l = 1; l <= L; ++l)
        if ((uint32_t)l > level) {
          const int32_t res = (int32_t)levelRes((uint32_t)l + 1);
#pragma unroll
          for (int a = 0; a < 3; ++a) {
            const int32_t id = clampToCell(oo[a], res);
            d.id[l][a]       = (uint32_t)id;
            d.tNext[l][a]    = planeT((float)(id + res * (int)(dirSign(d3[a]) >= 0)), g3[a], d.inv[a]);
          }
        }
    }
    bool left = true;
#pragma unroll
    for (int l = L - 1; l >= 0; --l)
      if (left && (uint32_t)l < level) {
        const uint32_t off = (d.id[l + 1][0] - d.id[l][0]) | (d.id[l + 1][1] - d.id[l][1]) |
                             (d.id[l + 1][2] - d.id[l][2]);
        left = off >= levelRes((uint32_t)l + 1);
        if (left)
          ddaStepCell(d, l);
      }
  }
};

// The same over a dense volume at depth 2 (the hit iterator's depth there).
struct DenseWalk {
  static constexpr int L = 2;
  f3 org, dir;
  DdaCell<L> d;
  float tMax;
  uint32_t budget;
  uint32_t node, leaf;  // unused

  __device__ __forceinline__ void query(const DevGrid &g, uint32_t attr, const DevValueRanges &vr, uint32_t &level,
                                        bool &empty)
  {
    level           = L;
    const float2 *p = DenseCellRanges<L>(g, attr).at(d.id[L][0], d.id[L][1], d.id[L][2]);
    empty           = true;
    if (p) {
      const float2 r = __ldg(p);
      empty          = !rangesOverlap(vr, r.x, r.y);
    }
  }
  __device__ __forceinline__ void step(uint32_t) { ddaStep(d); }
};

// intervalInit for a walk; returns nominalDeltaT.
template <class Walk>
__device__ __forceinline__ float walkInit(const DevGrid &g, f3 origin, f3 direction, float tLo, float tHi, Walk &w)
{
  IntervalItT<DdaCell<Walk::L>> it;
  it.dda = DdaCell<Walk::L>{};
  intervalInit(g, Walk::L, origin, direction, tLo, tHi, it);
  f3 org   = xfmPoint(g.objectToIndex, origin);
  w.org    = {org.x - (float)g.rootOrigin[0], org.y - (float)g.rootOrigin[1], org.z - (float)g.rootOrigin[2]};
  w.dir    = xfmVector(g.objectToIndex, direction);
  w.d      = it.dda;
  w.tMax   = it.tMax;
  w.budget = it.budget;
  w.node   = ~0u;
  w.leaf   = 0;
  return it.nominalDeltaT;
}

// One turn of intervalNext's loop.
template <class Walk>
__device__ __forceinline__ WalkResult walkStep(const DevGrid &g, uint32_t attr, const DevValueRanges &vr, Walk &w,
                                               float &t0, float &t1)
{
  if (!(w.d.t <= w.tMax))
    return kWalkEnd;
  uint32_t level = 0;
  bool empty     = true;
  w.query(g, attr, vr, level, empty);
  if (!empty) {
    if (!(w.d.t < w.tMax))
      return kWalkEnd;
    t0 = w.d.t;
  }
  if (w.budget-- == 0)
    return kWalkEnd;
  w.step(level);
  if (empty)
    return kWalkEmpty;
  t1 = minx(w.d.t, w.tMax);
  return kWalkInterval;
}

enum HitPhase : int {
  kHpAdvance,      // needs the next interval
  kHpBegin,        // marches [curT0, curT1)
  kHpMarch,        // next march step
  kHpMarchSample,  // march sample arrived
  kHpStartSample,  // sample at the interval start arrived
  kHpNudgeSample,  // nudged march sample arrived
  kHpBisectSample, // bisection sample arrived
  // phases of the state machine (no sample pending)
  kHpStartNudge,   // NaN start sample: nudge forward
  kHpMarchNudge,   // NaN march sample: nudge backward
  kHpValue,        // test value i
  kHpBisect,       // next bisection step
  kHpValueTail,    // end-point test of value i
  kHpRayDone,
  kHpNextRay,
  kHpDone
};

template <class Walk, class Field>
__global__ void __launch_bounds__(kBlock, kHitMinBlocks)
    kHitsWalk(const __grid_constant__ DevGrid g, uint32_t attr, DevValueRanges vr, uint32_t numValues,
              const float *__restrict__ values, uint64_t n, const float *__restrict__ orgs,
              const float *__restrict__ dirs, const float *__restrict__ tr, uint32_t maxPerRay,
              DevHit *__restrict__ outBase, uint32_t *__restrict__ counts)
{
  __shared__ float sv[kHitValues];
  const bool valuesShared = numValues <= kHitValues;
  if (valuesShared && threadIdx.x < numValues)
    sv[threadIdx.x] = __ldg(values + threadIdx.x);
  __syncthreads();
  Field F = [&]() {
    if constexpr (std::is_constructible<Field, const DevGrid &, uint32_t, uint32_t>::value)
      return Field(g, attr, kNumLevels - 1);
    else
      return Field(g, attr);
  }();
  // the warp's k-th ray: block k / 32 of its blocks, entry k % 32
  const uint64_t warps = (uint64_t)gridDim.x * (kBlock / 32);
  const uint64_t warp  = (uint64_t)blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5);
  const uint32_t below = (1u << (threadIdx.x & 31)) - 1u;
  uint64_t taken = 0, r = 0;

  Walk w;
  f3 o = {0.f, 0.f, 0.f}, dv = {0.f, 0.f, 0.f};
  uint32_t count = 0;
  int ph         = kHpDone;
  float step = 0.f, curT0 = 0.f, curT1 = 0.f, lastOffset = 0.f, cacheT = 0.f, cacheS = 0.f;
  // intersectBisection state
  float t0 = 0.f, s0 = 0.f, hs = 0.f, t = 0.f, s = 0.f, ts = 0.f;
  uint32_t march = 0, vi = 0;
  int nudge  = 0;
  float tHit = kPosInf, value = kPosInf, iso = 0.f;
  // bisect state
  float bt0 = 0.f, bs0 = 0.f, bt = 0.f, bs = 0.f, tol = 0.f, tMid = 0.f, tIso = kPosInf;
  int iter     = 0;
  float sample = 0.f, tReq = 0.f;

  ph = kHpNextRay;
  for (;;) {
    bool want           = false;
    const uint32_t idle = __ballot_sync(0xffffffffu, ph == kHpNextRay);
    if (idle) {
      if (ph == kHpNextRay) {
        const uint64_t k = taken + __popc(idle & below);
        r                = ((k >> 5) * warps + warp) * 32 + (k & 31);
        ph               = kHpDone;  // later rays of the warp are not below n either
        if (r < n) {
          o          = ld3(orgs, r);
          dv         = ld3(dirs, r);
          step       = walkInit(g, o, dv, __ldg(tr + 2 * r), __ldg(tr + 2 * r + 1), w);
          count      = 0;
          lastOffset = -kPosInf;
          cacheT     = __builtin_nanf("");
          cacheS     = 0.f;
          ph         = numValues ? kHpAdvance : kHpRayDone;
        }
      }
      taken += __popc(idle);
    }
    if (ph == kHpMarchSample) {
      // the sample of a march step: no isovalue within 1e-6 of either end
      // and none between them -> the next step (a superset of the exact
      // tests below, which decide everything else)
      s        = sample;
      cacheT   = t;
      cacheS   = s;
      bool any = isnan(s) || !valuesShared;
      if (valuesShared)
        for (uint32_t i = 0; i < numValues; ++i) {
          const float v = sv[i];
          any |= (fabsf(s0 - v) < 1e-6f) | (fabsf(s - v) < 1e-6f) | ((v - s0) * (v - s) < 0.f);
        }
      if (!any) {
        t0 = t;
        s0 = s;
        ++march;
        ph = kHpMarch;
      } else {
        ts    = t;
        nudge = 0;
        ph    = kHpMarchNudge;
      }
    } else if (ph == kHpStartSample) {
      s0 = sample;
      ph = kHpStartNudge;
    } else if (ph == kHpNudgeSample) {
      s  = sample;
      ph = kHpMarchNudge;
    } else if (ph == kHpBisectSample) {
      const float sm = sample;
      bool finished  = false;
      if (isnan(sm)) {
        tIso     = fabsf(iso - bs0) < fabsf(iso - bs) ? bt0 : bt;
        finished = true;
      } else if (sm == iso || (iso - bs0) * (iso - sm) < 0.f) {
        bt = tMid;
        bs = sm;
      } else if (bs == iso || (iso - bs) * (iso - sm) < 0.f) {
        bt0 = tMid;
        bs0 = sm;
      } else {
        tIso     = kPosInf;
        finished = true;
      }
      if (finished) {
        if (tIso < tHit && tIso <= curT1) {
          tHit  = tIso;
          value = iso;
        }
        ph = kHpValueTail;
      } else {
        ++iter;
        ph = kHpBisect;
      }
    }
    // the exact tests of a step, until a sample is needed or the step is done
    while (!want && ph >= kHpStartNudge && ph < kHpRayDone) {
      switch (ph) {
      case kHpStartNudge:
        if ((float)nudge < 10.f && isnan(s0) && t0 < curT1) {
          t0 += maxx(1e-5f, 1e-5f * step);
          ++nudge;
          tReq = t0;
          want = true;
          ph   = kHpStartSample;
        } else {
          ph = kHpMarch;
        }
        break;
      case kHpMarchNudge:
        if ((float)nudge < 10.f && isnan(s) && ts > t0) {
          ts -= maxx(1e-5f, 1e-5f * step);
          ++nudge;
          tReq = ts;
          want = true;
          ph   = kHpNudgeSample;
        } else {
          tHit  = kPosInf;
          value = kPosInf;
          vi    = 0;
          ph    = kHpValue;
        }
        break;
      case kHpValue:
        if (vi == numValues) {
          if (tHit < kPosInf) {
            const float eps = 0.125f * step;
            const DevHit hit{tHit, value, eps * sqrtf(dv.x * dv.x + dv.y * dv.y + dv.z * dv.z)};
            if (count < maxPerRay)
              outBase[r * maxPerRay + count] = hit;
            ++count;
            curT0      = hit.t + hit.epsilon;
            lastOffset = curT0;
            ph         = count >= kMaxHitsPerRay || curT0 == kPosInf ? kHpRayDone
                         : curT1 <= curT0                             ? kHpAdvance
                                                                      : kHpBegin;
          } else {
            t0 = t;
            s0 = s;
            ++march;
            ph = kHpMarch;
          }
          break;
        }
        iso = __ldg(values + vi);
        if (fabsf(s0 - iso) < 1e-6f) {
          if (t0 < tHit && t0 <= curT1) {
            tHit  = t0;
            value = iso;
          }
          ph = kHpValueTail;
        } else if (!isnan(s0 + s) && (iso - s0) * (iso - s) < 0.f) {
          bt0  = t0;
          bs0  = s0;
          bt   = ts;
          bs   = s;
          tol  = minx(1e-6f, 0.01f * hs);
          iter = 0;
          tMid = 0.f;
          ph   = kHpBisect;
        } else {
          ph = kHpValueTail;
        }
        break;
      case kHpBisect:
        if (iter < 10) {
          tMid              = 0.5f * (bt0 + bt);
          const float error = 0.5f * (bt - bt0);
          if (!(error < tol)) {
            tReq = tMid;
            want = true;
            ph   = kHpBisectSample;
            break;
          }
        }
        tIso = tMid;
        if (tIso < tHit && tIso <= curT1) {
          tHit  = tIso;
          value = iso;
        }
        ph = kHpValueTail;
        break;
      default:  // kHpValueTail
        if (t == curT1 && fabsf(s - iso) < 1e-6f) {
          if (ts < tHit && ts <= curT1) {
            tHit  = ts;
            value = iso;
          }
        }
        ++vi;
        ph = kHpValue;
        break;
      }
    }
    if (ph == kHpMarch) {
      if (t0 < curT1 && march < kMaxMarchSteps) {
        hs   = minx(step, curT1 - t0);
        t    = t0 + hs;
        tReq = t;
        want = true;
        ph   = kHpMarchSample;
      } else {
        ph = kHpAdvance;  // interval exhausted without a hit
      }
    }
    if (ph == kHpRayDone) {
      counts[r] = count;
      ph        = kHpNextRay;
    }
    if (ph == kHpAdvance) {
      float a = 0.f, b = 0.f;
      const WalkResult res = walkStep(g, attr, vr, w, a, b);
      if (res == kWalkEnd) {
        ph = kHpRayDone;
      } else if (res == kWalkInterval) {
        a = maxx(a, lastOffset);
        if (!(b <= a)) {
          curT0 = a;
          curT1 = b;
          ph    = kHpBegin;
        }
      }
    }
    if (ph == kHpBegin) {
      t0    = curT0;
      nudge = 0;
      march = 0;
      if (t0 == cacheT) {
        s0 = cacheS;
        ph = isnan(s0) ? kHpStartNudge : kHpMarch;
        if (ph == kHpMarch && t0 < curT1) {
          hs   = minx(step, curT1 - t0);
          t    = t0 + hs;
          tReq = t;
          want = true;
          ph   = kHpMarchSample;
        }
      } else {
        tReq = t0;
        want = true;
        ph   = kHpStartSample;
      }
    }
    if (__any_sync(0xffffffffu, want)) {
      if (want)
        sample = sampleLinear(F, xfmPoint(g.objectToIndex, f3{o.x + tReq * dv.x, o.y + tReq * dv.y,
                                                              o.z + tReq * dv.z}));
    } else if (!__any_sync(0xffffffffu, ph != kHpDone)) {
      return;
    }
  }
}

inline unsigned blocksFor(uint64_t n) { return (unsigned)((n + kBlock - 1) / kBlock); }

}  // namespace

void launchHits(const DevGrid &g, uint32_t attr, int filter, uint32_t depth, DevValueRanges vr,
                uint32_t numValues, const float *values, uint64_t n, const float *origins,
                const float *directions, const float *tRanges, uint32_t maxPerRay, DevHit *out,
                uint32_t *counts, cudaStream_t st)
{
  if (!n)
    return;
  auto walk = [&](auto kernel) {
    // persistent: as many CTAs as are resident at once
    int dev = 0, sms = 0, perSM = 0;
    cudaCheck(cudaGetDevice(&dev), "cudaGetDevice");
    cudaCheck(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "attribute");
    cudaCheck(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, kernel, kBlock, 0), "occupancy");
    const unsigned grid = (unsigned)std::min<uint64_t>(blocksFor(n), (uint64_t)sms * (uint64_t)std::max(perSM, 1));
    kernel<<<grid, kBlock, 0, st>>>(g, attr, vr, numValues, values, n, origins, directions, tRanges, maxPerRay, out,
                                    counts);
  };
  const bool mapped = leafMapApplies(g, kNumLevels - 1);
  auto sparse       = [&](auto tag) {
    using T = decltype(tag);
    if (mapped)
      walk(kHitsWalk<SparseWalk, MappedField<T>>);
    else
      walk(kHitsWalk<SparseWalk, SparseField<T>>);
  };
  if (filter != kFilterLinear || g.type[attr] != kFloat || g.temporal || (g.dense ? depth != 2 : depth < 3)) {
    launchHitsAny(g, attr, filter, depth, vr, numValues, values, n, origins, directions, tRanges, maxPerRay, out,
                  counts, st);
    return;
  }
  if (g.dense) {
    walk(kHitsWalk<DenseWalk, DenseField<float>>);
  } else {
    switch (g.compress) {
    case kCompressFP16Blocks:
      sparse(Blocked<CodeFP16>{});
      break;
    case kCompressBF16Blocks:
      sparse(Blocked<CodeBF16>{});
      break;
    case kCompressFP8Blocks:
      sparse(Blocked<CodeE4M3>{});
      break;
    case kCompressFP16:
      sparse(CodeFP16{});
      break;
    case kCompressBF16:
      sparse(CodeBF16{});
      break;
    case kCompressFP8:
      sparse(CodeE4M3{});
      break;
    default:
      sparse(float{});
    }
  }
  cudaCheck(cudaGetLastError(), "hit kernel launch");
}

}  // namespace vklcuda
