// Photon transport kernels for sm_100a.
//
// One persistent kernel runs the whole GGEMS photon loop for every history:
// primary generation (X-ray cone or voxelized source), FindSolid /
// ProjectToSolid over all solids, and the per-step tracking through the
// current solid (voxelized phantom or CT detector box), with Compton,
// photoelectric and Rayleigh sampling from GGEMS's tables and the dose /
// histogram tallies.  It replaces the reference's host loop of
// 2*S+2 launches per iteration (src/global/GGEMS.cc:303-363,
// src/navigators/GGEMSNavigator.cc:320-530) and its is_alive round trip.
//
// Design:
//  * each lane owns one random slot (JKISS state in registers) and runs that
//    slot's histories in batch order, so every history draws exactly the
//    random numbers the reference's slot would; lanes fetch slots from a
//    device work counter;
//  * a lane takes up to kTrackSteps voxel steps that need no logarithm (the
//    draws show that the photon crosses its voxel), or one part of anything else
//    (a whole step, an interaction, a FindSolid/ProjectToSolid round) per loop
//    iteration, and starts its next history as soon as one ends, so lanes never
//    idle while others finish long histories;
//  * the per-navigator cross-section tables (float4 per material and energy
//    bin), energy bins and photon cuts are staged into shared memory with
//    cp.async.bulk completing on an mbarrier (bounded wait);
//  * tallies: int32 histogram counts, int64 fixed-point energy deposits
//    (order independent), double energy^2.
//
// Arithmetic follows the reference operation by operation in float (double
// where it uses double) and the file is compiled with -fmad=false so that no
// multiply-add is contracted; the CPU oracle does the same.
#include <cfloat>
#include <cstdint>
#include <type_traits>

#include "gg_internal.cuh"

namespace gg {
namespace {

constexpr float kTwoPi = 6.283185307179586f;             // GGEMSConstants.hh:39
constexpr float kElectronMassC2 = 0.510998910f;           // GGEMSConstants.hh:52
constexpr float kTolerance = 5.0e-04f;                    // GGEMSGeometryConstants.hh:39
constexpr float kEps6 = 1.0e-06f;                         // GGEMSGeometryConstants.hh:38
constexpr float kOutOfWorld = FLT_MAX;                    // GGEMSParticleConstants.hh:44
constexpr int kNoProcess = 99;
constexpr float kRayleighFactor = 32526509815670243328.0f;  // GGEMSRayleighScatteringModels.hh:36
// KissUniform's (float)((double)x / 4294967295.0 * (1 - 2^-23)) equals, for
// every float x = (float)(uint32), the single-precision fused multiply-add
// fma(x, kKissCorrection, x * 2^-32): x * 2^-32 is exact and
// x * kKissCorrection + x * 2^-32 = x * 2^-32 * (1 - 2^-23 + 2^-32) is rounded
// once, which lands on the same float as the reference's double arithmetic for
// all 83,886,080 such x (checked exhaustively in tests/test_rng.py, against
// the division and against the double product).
constexpr float kKissTwoToMinus32 = 0x1p-32f;
constexpr float kKissCorrection = -0x1.ffp-56f;  // -(2^-23 - 2^-32) * 2^-32, exact in float

// Tracking steps a lane takes between two looks at its warp's waiting photons.
// The look (ballots, counts, the stash's exchange test) costs every lane more
// than a step; a lane that stops early idles for the rest.  8 / 12 / 16 / 20 / 24
// steps, the better of two runs: CBCT of 1e8 primaries 165.6 / 165.3 / 160.0 /
// 156.7 / 155.5 ms, 36 projections of 1e6 27.2 / 26.2 / 26.0 / 25.2 / 24.6 ms, 64^3
// dose of 1e6 1.66 / 1.67 / 1.65 / 1.62 / 1.63 ms; the two runs of one differ by up
// to 5 %, so 16 and more are alike.
constexpr int kTrackSteps = 16;
constexpr float kTwo23 = 8388608.0f;

// kTrackVoxel: steps of a voxelized solid that surely cross their voxel.
// kInteract: any other step of a voxelized solid, any step of a detector box, or
// the Compton / Rayleigh part of a meshed solid's step.
enum Phase : int { kNewHistory = 0, kFind = 1, kTrackVoxel = 2, kTrackMesh = 4, kInteract = 5, kDone = 6 };

struct V3 {
  float x, y, z;
};
__device__ __forceinline__ V3 v3(float x, float y, float z) { return V3{x, y, z}; }
__device__ __forceinline__ V3 add(V3 a, V3 b) { return v3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ V3 sub(V3 a, V3 b) { return v3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ V3 mul(V3 a, V3 b) { return v3(a.x * b.x, a.y * b.y, a.z * b.z); }
__device__ __forceinline__ V3 divv(V3 a, V3 b) { return v3(a.x / b.x, a.y / b.y, a.z / b.z); }
__device__ __forceinline__ V3 scale(V3 a, float s) { return v3(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ float dot3(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ V3 normalize3(V3 v) { return scale(v, 1.0f / sqrtf(dot3(v, v))); }

// GGfloat44 (row-major) products, GGEMSMatrixOperations.hh:46-125.
__device__ __forceinline__ V3 m_point(const float* m, V3 p) {
  return v3(m[0] * p.x + m[1] * p.y + m[2] * p.z + m[3] * 1.0f, m[4] * p.x + m[5] * p.y + m[6] * p.z + m[7] * 1.0f,
            m[8] * p.x + m[9] * p.y + m[10] * p.z + m[11] * 1.0f);
}
__device__ __forceinline__ V3 m33(const float* m, V3 p) {
  return v3(m[0] * p.x + m[1] * p.y + m[2] * p.z, m[4] * p.x + m[5] * p.y + m[6] * p.z, m[8] * p.x + m[9] * p.y + m[10] * p.z);
}
__device__ __forceinline__ V3 m33t(const float* m, V3 p) {
  return v3(m[0] * p.x + m[4] * p.y + m[8] * p.z, m[1] * p.x + m[5] * p.y + m[9] * p.z, m[2] * p.x + m[6] * p.y + m[10] * p.z);
}
// GGEMSReferentialTransformation.hh:80-141
__device__ __forceinline__ V3 g2l_pos(const float* m, V3 p) { return m33t(m, v3(p.x - m[3], p.y - m[7], p.z - m[11])); }
__device__ __forceinline__ V3 l2g_pos(const float* m, V3 p) { return m_point(m, p); }
__device__ __forceinline__ V3 g2l_dir(const float* m, V3 d) { return normalize3(m33t(m, d)); }
__device__ __forceinline__ V3 l2g_dir(const float* m, V3 d) { return normalize3(m33(m, d)); }

// RotateUnitZ, GGEMSReferentialTransformation.hh:44-70
__device__ __forceinline__ V3 rotate_uz(V3 v, V3 u) {
  float up = u.x * u.x + u.y * u.y;
  if (up > 0) {
    up = sqrtf(up);
    float px = v.x, py = v.y, pz = v.z;
    v.x = (u.x * u.z * px - u.y * py) / up + u.x * pz;
    v.y = (u.y * u.z * px + u.x * py) / up + u.y * pz;
    v.z = -up * px + u.z * pz;
  } else if (u.z < 0.0f) {
    v.x = -v.x;
    v.z = -v.z;
  }
  return v;
}

// BinarySearch / LinearInterpolation, GGEMSMathAlgorithms.hh:46-86
__device__ __forceinline__ int binary_search(float key, const float* a, int size) {
  int low = 0, high = size - 1;
#pragma unroll 1
  while (high - low > 1) {
    int mid = (high + low) / 2;
    float v = a[mid];
    if (v == key) return mid;
    if (v < key) low = mid;
    else high = mid;
  }
  return low;
}
__device__ __forceinline__ float lerp_ref(float xa, float ya, float xb, float yb, float x) {
  if (xa > xb) return yb;
  if (xa >= x) return ya;
  if (xb <= x) return yb;
  return ya + (x - xa) * (yb - ya) / (xb - xa);
}

// Ray tracing, GGEMSRayTracing.hh:60-326
__device__ __forceinline__ float safety_in(float p, float mn, float mx) {
  float a = fabsf(p - mn), b = fabsf(p - mx);
  p = (a < kTolerance) ? mn + kTolerance : p;
  return (b < kTolerance) ? mx - kTolerance : p;
}
__device__ __forceinline__ float safety_out(float p, float mn, float mx) {
  float a = fabsf(p - mn), b = fabsf(p - mx);
  p = (a < kTolerance) ? mn - kTolerance : p;
  return (b < kTolerance) ? mx + kTolerance : p;
}
__device__ __forceinline__ V3 safety_inside(V3 p, V3 mn, V3 mx) {
  return v3(safety_in(p.x, mn.x, mx.x), safety_in(p.y, mn.y, mx.y), safety_in(p.z, mn.z, mx.z));
}
__device__ __forceinline__ V3 safety_outside(V3 p, V3 mn, V3 mx) {
  return v3(safety_out(p.x, mn.x, mx.x), safety_out(p.y, mn.y, mx.y), safety_out(p.z, mn.z, mx.z));
}
__device__ __forceinline__ bool in_aabb(V3 p, V3 mn, V3 mx) {
  if (p.x < (mn.x + kTolerance) || p.x > (mx.x - kTolerance)) return false;
  if (p.y < (mn.y + kTolerance) || p.y > (mx.y - kTolerance)) return false;
  if (p.z < (mn.z + kTolerance) || p.z > (mx.z - kTolerance)) return false;
  return true;
}
// inv holds 1.0f / d per axis (used only where |d| >= 1e-6, as the reference
// computes it there), so a direction's reciprocals can be computed once.
// The reference's early returns all give kOutOfWorld and its running
// tmin <= tmax test can only fail for good (tmin grows, tmax shrinks), so the
// axes are combined without branches and tested once at the end.
__device__ __forceinline__ float distance_to_aabb(V3 p, V3 d, V3 inv, V3 mn, V3 mx) {
  float tmin = FLT_MIN, tmax = FLT_MAX;
  bool miss = false;
  {
    const float a = (mn.x - p.x) * inv.x, b = (mx.x - p.x) * inv.x;
    const bool along = fabsf(d.x) < kEps6;
    miss = along && (p.x < mn.x || p.x > mx.x);
    tmin = along ? tmin : fminf(a, b);
    tmax = along ? tmax : fmaxf(a, b);
  }
  {
    const float a = (mn.y - p.y) * inv.y, b = (mx.y - p.y) * inv.y;
    const bool along = fabsf(d.y) < kEps6;
    miss = miss || (along && (p.y < mn.y || p.y > mx.y));
    tmin = along ? tmin : fmaxf(tmin, fminf(a, b));
    tmax = along ? tmax : fminf(tmax, fmaxf(a, b));
  }
  {
    const float a = (mn.z - p.z) * inv.z, b = (mx.z - p.z) * inv.z;
    const bool along = fabsf(d.z) < kEps6;
    miss = miss || (along && (p.z < mn.z || p.z > mx.z));
    tmin = along ? tmin : fmaxf(tmin, fminf(a, b));
    tmax = along ? tmax : fminf(tmax, fmaxf(a, b));
  }
  miss = miss || tmin > tmax || (tmin < 0.0f && tmax <= 0.0f);
  // the reference compares in double; 2 x kTolerance is exact in float
  miss = miss || (tmax - tmin) < 2.0f * kTolerance;
  const float t = tmin <= kEps6 ? tmax : tmin;
  return miss ? kOutOfWorld : t;
}

// Along a face (|d| < 1e-6) the reciprocal is infinite: distance_to_aabb does
// not read it there, and in the voxel step a face so far away never is the nearest.
__device__ __forceinline__ float reciprocal(float d) { return fabsf(d) < kEps6 ? __int_as_float(0x7f800000) : 1.0f / d; }
__device__ __forceinline__ V3 reciprocal(V3 d) { return v3(reciprocal(d.x), reciprocal(d.y), reciprocal(d.z)); }
__device__ __forceinline__ float distance_to_aabb(V3 p, V3 d, V3 mn, V3 mx) {
  return distance_to_aabb(p, d, reciprocal(d), mn, mx);
}

// JKISS32, GGEMSKissEngine.hh:50-75
__device__ __forceinline__ float kiss_uniform(float x) { return __fmaf_rn(x, kKissCorrection, x * kKissTwoToMinus32); }
struct Kiss {
  uint32_t s1, s2, s3, s4, s5;
  // the draw as a float in [0, 2^32]
  __device__ __forceinline__ float raw() {
    s2 ^= (s2 << 5);
    s2 ^= (s2 >> 7);
    s2 ^= (s2 << 22);
    int t = static_cast<int>(s3 + s4 + s5);
    s3 = s4;
    s5 = t < 0;
    s4 = static_cast<uint32_t>(t) & 2147483647u;
    s1 += 1411392427u;
    return __uint2float_rn(s1 + s2 + s4);
  }
  __device__ __forceinline__ float uniform() { return kiss_uniform(raw()); }
};

struct Photon {
  V3 p, d;          // global outside solids, local while tracking inside one
  float E;
  float psd;        // particle_solid_distance_
  int solid_id;
  int8_t status;
  int8_t scatter;
};

// Tables (shared memory when they fit, otherwise the HBM blob).
struct Tab {
  const unsigned char* base;
  const DevNavigator* nav;
  __device__ __forceinline__ const float* energy_bins(int n) const {
    return reinterpret_cast<const float*>(base + nav[n].energy_bins_offset);
  }
  __device__ __forceinline__ const float4* sigma(int n) const {
    return reinterpret_cast<const float4*>(base + nav[n].sigma_offset);
  }
  __device__ __forceinline__ const float* photon_cut(int n) const {
    return reinterpret_cast<const float*>(base + nav[n].photon_cut_offset);
  }
  // TLE tables: GG_ATTENUATION_BINS energies followed by mu_en per material
  __device__ __forceinline__ const float* attenuation(int n) const {
    return reinterpret_cast<const float*>(base + nav[n].attenuation_offset);
  }
};

__device__ __forceinline__ float pick(float4 s, int i) { return i == 0 ? s.x : (i == 1 ? s.y : s.z); }

// a / b correctly rounded from y = the correctly rounded 1 / b, without the
// division instruction sequence's branch to its slow path: one refinement makes
// the quotient faithful, the second is Markstein's final step (P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor",
// IBM J. Res. Dev. 34 (1990): a faithful q and a correctly rounded y give
// RN(q + y RN(a - b q)) = RN(a / b)).  Needs exponents away from the ends of the
// range.  The voxel step's are: b a voxel size of 8e-3 to 2048 mm, a a position of
// 5e-4 to 2048 mm above the border (fast_steps in gg_runtime.cu).
__device__ __forceinline__ float quotient(float a, float b, float y) {
  float q = a * y;
  q = __fmaf_rn(__fmaf_rn(-q, b, a), y, q);
  return __fmaf_rn(__fmaf_rn(-q, b, a), y, q);
}

// The draws of one GetPhotonNextInteraction call before their conversion to
// (0, 1): one per process, in process order (0 where a process is missing).
// three: every navigator of the launch has all three processes.
struct Draws {
  float x0, x1, x2;
};
__device__ __forceinline__ Draws draw_processes(Kiss& rng, uint32_t process_pack, bool three) {
  Draws w{0.0f, 0.0f, 0.0f};
  if (three) {
    w.x0 = rng.raw();
    w.x1 = rng.raw();
    w.x2 = rng.raw();
    return w;
  }
  const int n = static_cast<int>(process_pack & kPackCount);
  if (n > 0) w.x0 = rng.raw();
  if (n > 1) w.x1 = rng.raw();
  if (n > 2) w.x2 = rng.raw();
  return w;
}

// True only if every process's sampled distance -logf(u) / sigma is at least
// `distance`, which most steps show without a logarithm or a division: with
// x = the draw of u (u <= x / 2^32), -log(u) >= 1 - u >= 1 - x / 2^32, so
// sigma distance + x / 2^32 < 1 is enough.  The scale's 2^-18 covers the
// roundings of the product (2^-23), of logf (1 ulp, taken as 2^-22) and of the
// quotient (2^-24); the limit's 2^11 those of the sum (at most 2^8).  False
// where the test cannot tell (an infinite or NaN product among them); about the
// share of the steps that interact (1 - u against -log(u): half a per cent more
// of them at sigma distance = 0.01).
constexpr float kCrossScale = 0x1.00004p+32f;
constexpr float kCrossLimit = 0x1p+32f - 0x1p+11f;
__device__ __forceinline__ bool surely_crosses(Draws w, float4 sigma, float distance) {
  const float reach = distance * kCrossScale;
  return __fmaf_rn(sigma.x, reach, w.x0) < kCrossLimit && __fmaf_rn(sigma.y, reach, w.x1) < kCrossLimit &&
         __fmaf_rn(sigma.z, reach, w.x2) < kCrossLimit;
}

// GetPhotonNextInteraction, GGEMSPhotonNavigator.hh:57-93, of these draws.
// Returns the distance, writes the process; sigma is the table's row of the
// material and the cached BinarySearch result (process order), process_pack the
// navigator's process count and ids (DevNavigator).  One logarithm and one
// division in a loop: it runs for few steps, and its code for many warps' sake
// has to be short (see the kernel's comment on its instruction footprint).
__device__ __forceinline__ float next_interaction(Draws w, uint32_t process_pack, float4 sigma, int& proc) {
  float nid = kOutOfWorld;
  proc = kNoProcess;
  const int n = static_cast<int>(process_pack & kPackCount);
#pragma unroll 1
  for (int i = 0; i < n; ++i) {
    const float dist = -logf(kiss_uniform(i == 0 ? w.x0 : (i == 1 ? w.x1 : w.x2))) / pick(sigma, i);
    if (dist < nid) {
      nid = dist;
      proc = static_cast<int>((process_pack >> (8 * (i + 1))) & 0xffu);
    }
  }
  return nid;
}

// 16-byte shared-memory (or global) loads of a struct's leading fields.
__device__ __forceinline__ float4 load4f(const void* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ int4 load4i(const void* p) { return *reinterpret_cast<const int4*>(p); }

// State handed to and returned by the (out-of-line) interaction samplers: the
// photon's energy and the polar angle.  Passed by value so that the photon and
// its random state stay in registers in the transport loop (a reference would
// force them into local memory).  What both samplers end with, the azimuth and
// the rotation into the photon's frame, is in scatter(), once for both: lanes of
// either kind run it together and its code is there once.
struct Interaction {
  float E;
  float cost, sint;
  Kiss rng;
  int outcome;
};
enum : int { kTurned = 0, kUnchanged = 1, kAbsorbed = 2 };

// KleinNishinaComptonSampleSecondaries, GGEMSComptonScatteringModels.hh:47-132
__device__ __noinline__ Interaction compton(Interaction in) {
  Kiss rng = in.rng;
  float E0 = in.E;
  float E0m = E0 / kElectronMassC2;
  float eps0 = 1.0f / (1.0f + 2.0f * E0m);
  float eps0sq = eps0 * eps0;
  float alpha1 = -logf(eps0);
  float alpha2 = alpha1 + 0.5f * (1.0f - eps0sq);
  float eps, epssq, onecost, sint2, greject, r3;
  int nloop = 0;
  do {
    ++nloop;
    if (nloop > 1000) {
      in.rng = rng;
      in.outcome = kUnchanged;
      return in;
    }
    float r1 = rng.uniform();
    float r2 = rng.uniform();
    r3 = rng.uniform();
    if (alpha1 > alpha2 * r1) {
      eps = expf(-alpha1 * r2);
      epssq = eps * eps;
    } else {
      epssq = eps0sq + (1.0f - eps0sq) * r2;
      eps = sqrtf(epssq);
    }
    onecost = (1.0f - eps) / (eps * E0m);
    sint2 = onecost * (2.0f - onecost);
    greject = 1.0f - eps * sint2 / (1.0f + epssq);
  } while (greject < r3);
  if (sint2 < 0.0f) sint2 = 0.0f;
  in.E = E0 * eps;
  in.cost = 1.0f - onecost;
  in.sint = sqrtf(sint2);
  in.rng = rng;
  return in;
}

__constant__ float c_rayleigh_pp[9][101];

__device__ __noinline__ float exp_minus_n_log(float n, float v) { return expf(-n * logf(v)); }
__device__ __noinline__ float rayleigh_w(float x, float n) {
  return (x < 0.02f) ? n * x * (1.0f - 0.5f * (n - 1.0f) * x * (1.0f - (n - 2.0f) * x / 3.0f))
                     : 1.0f - exp_minus_n_log(n, 1.0f + x);
}

// LivermoreRayleighSampleSecondaries, GGEMSRayleighScatteringModels.hh:169-316
__device__ __noinline__ Interaction rayleigh(Interaction in, const DevNavigator& nv, const float* ebins,
                                             const float4* sig, int material, int energy_id) {
  float E0 = in.E;
  if (E0 <= 250.0e-6f) {
    in.outcome = kAbsorbed;
    return in;
  }
  Kiss rng = in.rng;
  const int nb = nv.number_of_bins;
  int n_minus_one = static_cast<int8_t>(nv.number_of_elements[material] - 1);
  int mixture = nv.element_offset[material];
  int z = nv.atomic_number[mixture + n_minus_one];
  if (n_minus_one > 0) {
    const float4* row = sig + static_cast<size_t>(material * nb + energy_id);
    const int slot = nv.process_id[0] == GG_RAYLEIGH_SCATTERING ? 0 : (nv.process_id[1] == GG_RAYLEIGH_SCATTERING ? 1 : 2);
    float kcs = lerp_ref(ebins[energy_id], pick(row[0], slot), ebins[energy_id + 1], pick(row[1], slot), E0);
    float x = rng.uniform() * kcs;
    float cs = 0.0f;
#pragma unroll 1
    for (int i = 0; i < n_minus_one; ++i) {
      int zi = nv.atomic_number[mixture + i];
      const float* pa = nv.rayleigh_per_atom + nb * zi;
      cs += nv.atomic_number_density[mixture + i] *
            lerp_ref(ebins[energy_id], pa[energy_id], ebins[energy_id + 1], pa[energy_id + 1], E0);
      if (x < cs) {
        z = zi;
        break;
      }
    }
  }
  float xx = kRayleighFactor * E0 * E0;
  float n0 = c_rayleigh_pp[6][z] - 1.0f, n1 = c_rayleigh_pp[7][z] - 1.0f, n2 = c_rayleigh_pp[8][z] - 1.0f;
  float b0 = c_rayleigh_pp[3][z], b1 = c_rayleigh_pp[4][z], b2 = c_rayleigh_pp[5][z];
  float w0 = rayleigh_w(2.0f * xx * b0, n0);
  float w1 = rayleigh_w(2.0f * xx * b1, n1);
  float w2 = rayleigh_w(2.0f * xx * b2, n2);
  float x0 = w0 * c_rayleigh_pp[0][z] / (b0 * n0);
  float x1 = w1 * c_rayleigh_pp[1][z] / (b1 * n1);
  float x2 = w2 * c_rayleigh_pp[2][z] / (b2 * n2);
  float cost;
  do {
    float w = w0, n = n0, b = b0;
    float x = rng.uniform() * (x0 + x1 + x2);
    if (x > x0) {
      x -= x0;
      if (x <= x1) {
        w = w1; n = n1; b = b1;
      } else {
        w = w2; n = n2; b = b2;
      }
    }
    n = 1.0f / n;
    float y = rng.uniform() * w;
    if (y < 0.02f) x = y * n * (1.0f + 0.5f * (n + 1.0f) * y * (1.0f - (n + 2.0f) * y / 3.0f));
    else x = exp_minus_n_log(n, 1.0f - y) - 1.0f;
    cost = 1.0f - x / (b * xx);
  } while (2.0f * rng.uniform() > 1.0f + cost * cost || cost < -1.0f);
  in.cost = cost;
  in.sint = sqrtf((1.0f - cost) * (1.0f + cost));
  in.rng = rng;
  return in;
}

// Compton or Rayleigh interaction of the photon (proc is one of the two).
__device__ __forceinline__ void scatter(Photon& ph, Kiss& rng, int proc, const DevNavigator& nv, const float* ebins,
                                        const float4* sig, int material, int energy_id) {
  Interaction in{ph.E, 0.0f, 0.0f, rng, kTurned};
  in = proc == GG_COMPTON_SCATTERING ? compton(in) : rayleigh(in, nv, ebins, sig, material, energy_id);
  ph.E = in.E;
  rng = in.rng;
  if (in.outcome == kTurned) {
    const float phi = rng.uniform() * kTwoPi;
    float sin_phi, cos_phi;
    sincosf(phi, &sin_phi, &cos_phi);  // the same bits as sinf and cosf
    ph.d = normalize3(rotate_uz(v3(in.sint * cos_phi, in.sint * sin_phi, in.cost), ph.d));
  }
  if (in.outcome == kAbsorbed) ph.status = GG_DEAD;
}

// dose_record_standard / dose_photon_tracking, GGEMSDoseRecording.hh:65-118
__device__ __forceinline__ int dosel(const DevDoseMap& dm, V3 p) {
  if (p.x < dm.border_min[0] + kEps6 || p.x > dm.border_max[0] - kEps6) return -1;
  if (p.y < dm.border_min[1] + kEps6 || p.y > dm.border_max[1] - kEps6) return -1;
  if (p.z < dm.border_min[2] + kEps6 || p.z > dm.border_max[2] - kEps6) return -1;
  int ix = __float2int_rz((p.x - dm.border_min[0]) * dm.inv_size_of_dosels[0]);
  int iy = __float2int_rz((p.y - dm.border_min[1]) * dm.inv_size_of_dosels[1]);
  int iz = __float2int_rz((p.z - dm.border_min[2]) * dm.inv_size_of_dosels[2]);
  if (ix < 0 || ix >= dm.number_of_dosels[0]) return -1;
  if (iy < 0 || iy >= dm.number_of_dosels[1]) return -1;
  if (iz < 0 || iz >= dm.number_of_dosels[2]) return -1;
  return ix + iy * dm.number_of_dosels[0] + iz * dm.number_of_dosels[0] * dm.number_of_dosels[1];
}
__device__ __forceinline__ void dose_record(const DevDoseMap& dm, float edep, V3 p) {
  int id = dosel(dm, p);
  if (id < 0) return;
  if (dm.hit) atomicAdd(dm.hit + id, 1);
  long long q = __double2ll_rn(static_cast<double>(edep) * kEdepScale);
  atomicAdd(dm.edep + id, static_cast<unsigned long long>(q));
  if (dm.edep_squared) atomicAdd(dm.edep_squared + id, static_cast<double>(edep) * static_cast<double>(edep));
}

// A new primary, get_primaries_ggems_xray_source (GetPrimariesGGEMSXRaySource.cl:52-143)
// or get_primaries_ggems_voxelized_source (GetPrimariesGGEMSVoxelizedSource.cl:57-150):
// both start with the cone angles and end with the energy, so one copy of that
// code serves both.  Out of line (it runs once per history, in the warp's rare
// round): keeps its FP64 cone sampling out of the tracking loop's
// instruction footprint; state in and out by value, so nothing goes to the
// stack.  Measured +0.8 % on the CBCT projection.
struct PrimaryOut {
  V3 p, d;
  float E;
  Kiss rng;
};
__device__ __noinline__ PrimaryOut new_primary(Kiss rng, const DevSource& s) {
  PrimaryOut out;
  const bool xray = s.type == GG_SOURCE_XRAY;
  double phi = rng.uniform();
  double theta = rng.uniform();
  phi *= static_cast<double>(kTwoPi);
  theta = acos(1.0 - (xray ? s.new_aperture : 2.0) * theta);
  double st, ct, sp, cp;  // sincos gives the same bits as sin and cos
  sincos(theta, &st, &ct);
  sincos(phi, &sp, &cp);
  const V3 rot = v3(static_cast<float>(cp * st), static_cast<float>(sp * st), static_cast<float>(ct));
  V3 p;
  if (xray) {
    p = l2g_pos(s.matrix, v3(0.0f, 0.0f, 0.0f));
    const V3 dir = normalize3(sub(v3(0.0f, 0.0f, 0.0f), p));
    out.d = normalize3(rotate_uz(rot, dir));
    p.x = s.focal_spot_size[0] * (rng.uniform() - 0.5f);
    p.y = s.focal_spot_size[1] * (rng.uniform() - 0.5f);
    p.z = s.focal_spot_size[2] * (rng.uniform() - 0.5f);
  } else {
    out.d = rot;
    const float rnd_act = rng.uniform();
    const int ia = binary_search(rnd_act, s.activity_cdf, s.number_of_activity_bins);
    const int vox = s.activity_index[ia];
    const int nx = s.number_of_voxels[0], slice = nx * s.number_of_voxels[1];
    const int iz = vox / slice, in_slice = vox - iz * slice;
    const int iy = in_slice / nx, ix = in_slice - iy * nx;
    const V3 bmin = v3(s.border_min[0], s.border_min[1], s.border_min[2]);
    const V3 vs = v3(s.voxel_sizes[0], s.voxel_sizes[1], s.voxel_sizes[2]);
    const V3 vmin = add(bmin, mul(v3(static_cast<float>(ix), static_cast<float>(iy), static_cast<float>(iz)), vs));
    p.x = bmin.x + (static_cast<float>(ix) + rng.uniform()) * vs.x;
    p.y = bmin.y + (static_cast<float>(iy) + rng.uniform()) * vs.y;
    p.z = bmin.z + (static_cast<float>(iz) + rng.uniform()) * vs.z;
    p = safety_inside(p, vmin, add(vmin, vs));
  }
  out.p = l2g_pos(s.matrix, p);
  int index = 0;
  float rnd = 0.0f;
  if (s.number_of_energy_bins != 1) {
    rnd = rng.uniform();
    index = binary_search(rnd, s.energy_cdf, s.number_of_energy_bins + 1);
  }
  out.E = !s.is_interp ? s.energy_spectrum[index]
                       : lerp_ref(s.energy_cdf[index], s.energy_spectrum[index], s.energy_cdf[index + 1],
                                  s.energy_spectrum[index + 1], rnd);
  out.rng = rng;
  return out;
}

// Track-length-estimator deposit of one voxel step
// (TrackThroughGGEMSVoxelizedSolid.cl:286-301): E * mu_en(E, material) * step
// (mm -> cm), with mu_en interpolated in the 220-bin attenuation table.
// e_index: the energy's bin there, which a photon keeps between interactions:
// searched once per run of steps, not per step.
__device__ __forceinline__ float tle_edep(const float* att, int material, int e_index, float energy, float step) {
  const float* me = att + GG_ATTENUATION_BINS * (1 + material);
  float mu_en = e_index == 0 ? me[0] : lerp_ref(att[e_index - 1], me[e_index - 1], att[e_index], me[e_index], energy);
  return energy * mu_en * step * 0.1f;
}

// ---- meshed solid (TrackThroughGGEMSMeshSolid.cl) ----
constexpr int kMaxMeshCrossings = 16;  // MAX_TRIANGLE_INTERACTION

struct MeshCrossings {
  V3 first, second;  // nearest and second nearest crossing
  int count;
};

__device__ __forceinline__ V3 cross3(V3 a, V3 b) {
  return v3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}

// GetMeshIOPositions (l.249-318): every octree node that owns triangles, in
// node order, is slab-tested (TestLineNode, l.182-230, with the direction's
// reciprocals) and its triangles are intersected with the Moller-Trumbore test
// (l.121-170).  GGEMS keeps up to 16 crossings sorted by squared distance (a
// new crossing goes after equal ones) but only reads the first two, so only
// those two are kept here, with the same ordering rule; the search ends at 16
// crossings (GGEMS writes past its array beyond that).
// Moller-Trumbore test of triangle k (l.121-170) and GGEMS's crossing
// ordering: a new crossing goes before the kept ones only when strictly
// nearer (squared distance, l.276-303).  Returns true once 16 crossings were
// counted.
struct CrossingState {
  float d0, d1;
  bool have0, have1;
};
__device__ __forceinline__ bool add_crossing(V3 p, V3 d, const float4* tris, int k, MeshCrossings& out, CrossingState& c) {
  const float4 t0 = __ldg(tris + 3 * k), t1 = __ldg(tris + 3 * k + 1), t2 = __ldg(tris + 3 * k + 2);
  const V3 p0 = v3(t0.x, t0.y, t0.z), e1 = v3(t0.w, t1.x, t1.y), e2 = v3(t1.z, t1.w, t2.x);
  const V3 h = cross3(d, e2);
  const float det = dot3(e1, h);
  if (det > -kEps6 && det < kEps6) return false;
  const float f = 1.0f / det;
  const V3 sv = sub(p, p0);
  const float u = f * dot3(sv, h);
  if (u < 0.0f || u > 1.0f) return false;
  const V3 q = cross3(sv, e1);
  const float v = f * dot3(q, d);
  if (v < 0.0f || u + v > 1.0f) return false;
  const float t = f * dot3(q, e2);
  if (!(t > kEps6)) return false;
  const V3 x = v3(p.x + d.x * t, p.y + d.y * t, p.z + d.z * t);
  const float dx = x.x - p.x, dy = x.y - p.y, dz = x.z - p.z;
  const float d2 = dx * dx + dy * dy + dz * dz;
  if (!c.have0 || d2 < c.d0) {
    if (c.have0) {
      out.second = out.first;
      c.d1 = c.d0;
      c.have1 = true;
    }
    out.first = x;
    c.d0 = d2;
    c.have0 = true;
  } else if (!c.have1 || d2 < c.d1) {
    out.second = x;
    c.d1 = d2;
    c.have1 = true;
  }
  return ++out.count == kMaxMeshCrossings;
}

// Slab test of the ray [0, inf) against a box (TestLineNode, l.182-230).
__device__ __forceinline__ bool ray_hits_box(const float pos[3], const float dir[3], const float ood[3],
                                             const float mn[3], const float mx[3]) {
  float tmin = 0.0f, tmax = FLT_MAX;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    if (fabsf(dir[i]) < kEps6) {
      if (pos[i] < mn[i] || pos[i] > mx[i]) return false;
    } else {
      float t1 = (mn[i] - pos[i]) * ood[i], t2 = (mx[i] - pos[i]) * ood[i];
      if (t1 > t2) {
        float t = t2;
        t2 = t1;
        t1 = t;
      }
      if (t1 > tmin) tmin = t1;
      if (t2 < tmax) tmax = t2;
      if (tmin > tmax) return false;
    }
  }
  return true;
}

// GetMeshIOPositions (l.249-318).  GGEMS keeps up to 16 crossings sorted by
// squared distance but only reads the first two and the count (whose parity
// says inside / outside), so only those are kept here, with the same ordering
// rule; the search ends at 16 crossings (GGEMS writes past its array beyond
// that).  Octree form: every node that owns triangles, in node order, is
// slab-tested and its triangles intersected, exactly GGEMS's scan.  BVH form
// (large meshes): a hierarchy of four children a node is walked in order with a
// stack; each triangle test is the same arithmetic, so the crossings found are
// the same set and only their discovery order (hence exact ties) can differ from
// the scan's.
__device__ __noinline__ MeshCrossings mesh_crossings(V3 p, V3 d, V3 inv, const float4* nodes, int node_count,
                                                     const float4* tris, int bvh) {
  MeshCrossings out;
  out.count = 0;
  out.first = out.second = p;
  CrossingState c{FLT_MAX, FLT_MAX, false, false};
  const float dir[3] = {d.x, d.y, d.z}, pos[3] = {p.x, p.y, p.z}, ood[3] = {inv.x, inv.y, inv.z};
  if (!bvh) {
    for (int n = 0; n < node_count; ++n) {
      const float4 a = __ldg(nodes + 2 * n), b = __ldg(nodes + 2 * n + 1);
      const float mn[3] = {a.x, a.y, a.z}, mx[3] = {a.w, b.x, b.y};
      if (!ray_hits_box(pos, dir, ood, mn, mx)) continue;
      const int first = __float_as_int(b.z), count = __float_as_int(b.w);
      for (int k = first; k < first + count; ++k)
        if (add_crossing(p, d, tris, k, out, c)) return out;
    }
    return out;
  }
  // A lane walks down to its next leaf, then all lanes that have one test their
  // triangles together.  What bounds the walk is divergence (lanes leave it after
  // different numbers of nodes and leaves: 5 of 32 active) and the chain of node
  // loads.  Four boxes a node halve both against two children with a box tested
  // per step: 245,760 triangles, 1e7 primaries 80.5 -> 52.8 ms (under the
  // profiler 2e6 primaries 16.3 -> 10.5 ms, 22 % fewer warp instructions, issue
  // slots 52 -> 63 % busy).
  int stack[kMeshStack];
  int sp = 0, ref = 0;
  const bool along = fabsf(d.x) < kEps6 || fabsf(d.y) < kEps6 || fabsf(d.z) < kEps6;
  for (;;) {
    while (ref >= 0 && ref != kMeshNoChild) {
      const float4* n = nodes + static_cast<size_t>(kMeshNodeFloat4) * ref;
      const float4 lx = __ldg(n), hx = __ldg(n + 1), ly = __ldg(n + 2), hy = __ldg(n + 3), lz = __ldg(n + 4), hz = __ldg(n + 5);
      const int4 child = __ldg(reinterpret_cast<const int4*>(n + 6));
      auto hit = [&](float x0, float x1, float y0, float y1, float z0, float z1) -> bool {
        if (along) {
          const float mn[3] = {x0, y0, z0}, mx[3] = {x1, y1, z1};
          return ray_hits_box(pos, dir, ood, mn, mx);
        }
        // ray_hits_box without its tests for a direction along a face; its early
        // returns only save work (tmin grows, tmax shrinks)
        const float ax = (x0 - p.x) * inv.x, bx = (x1 - p.x) * inv.x, ay = (y0 - p.y) * inv.y, by = (y1 - p.y) * inv.y,
                    az = (z0 - p.z) * inv.z, bz = (z1 - p.z) * inv.z;
        const float tmin = fmaxf(fmaxf(fminf(ax, bx), fminf(ay, by)), fmaxf(fminf(az, bz), 0.0f));
        const float tmax = fminf(fminf(fmaxf(ax, bx), fmaxf(ay, by)), fminf(fmaxf(az, bz), FLT_MAX));
        return !(tmin > tmax);
      };
      // the first child hit is next, the others wait on the stack, the last one at the bottom
      int next = kMeshNoChild;
      if (hit(lx.w, hx.w, ly.w, hy.w, lz.w, hz.w)) next = child.w;
      if (hit(lx.z, hx.z, ly.z, hy.z, lz.z, hz.z)) {
        if (next != kMeshNoChild) stack[sp++] = next;
        next = child.z;
      }
      if (hit(lx.y, hx.y, ly.y, hy.y, lz.y, hz.y)) {
        if (next != kMeshNoChild) stack[sp++] = next;
        next = child.y;
      }
      if (hit(lx.x, hx.x, ly.x, hy.x, lz.x, hz.x)) {
        if (next != kMeshNoChild) stack[sp++] = next;
        next = child.x;
      }
      if (next == kMeshNoChild && sp > 0) next = stack[--sp];
      ref = next;
    }
    if (ref == kMeshNoChild) break;
    const int first = static_cast<int>(static_cast<uint32_t>(~ref) / kMeshLeaf);
    const int end = first + static_cast<int>(static_cast<uint32_t>(~ref) % kMeshLeaf) + 1;
#pragma unroll 1
    for (int k = first; k < end; ++k)
      if (add_crossing(p, d, tris, k, out, c)) return out;
    ref = sp > 0 ? stack[--sp] : kMeshNoChild;
  }
  return out;
}

// world_tracking (WorldTracking.cl:54-162): the flight from the photon's
// position to the solid FindSolid chose (10 m when none) sampled in steps of
// the world element size along the dominant axis.
__device__ __noinline__ void world_track(V3 p1, V3 dir, float E, float psd, const TransportParams& P) {
  float distance = psd == kOutOfWorld ? 10000.0f : psd;
  if (distance <= kTolerance) return;
  const V3 size = v3(P.world_sizes[0], P.world_sizes[1], P.world_sizes[2]);
  const int nx = P.world_dimensions[0], ny = P.world_dimensions[1], nz = P.world_dimensions[2];
  const V3 p2 = add(p1, scale(dir, distance));
  const V3 lo = v3(size.x * static_cast<float>(nx) * -0.5f, size.y * static_cast<float>(ny) * -0.5f,
                   size.z * static_cast<float>(nz) * -0.5f);
  V3 q = divv(sub(p1, lo), size);
  int ix = __float2int_rz(q.x), iy = __float2int_rz(q.y), iz = __float2int_rz(q.z);
  const V3 diff = sub(p2, p1);
  float length = fabsf(diff.x), main_size = size.x;
  if (fabsf(diff.y) > length) {
    length = fabsf(diff.y);
    main_size = size.y;
  } else if (fabsf(diff.z) > length) {
    length = fabsf(diff.z);
    main_size = size.z;
  }
  const float inv_length = 1.0f / length;
  const V3 increment = v3(inv_length * diff.x, inv_length * diff.y, inv_length * diff.z);
  const int steps = static_cast<int>(1.0f + (length / main_size));
  const size_t cells = static_cast<size_t>(nx) * ny * nz;
  const long long e_fixed = __double2ll_rn(static_cast<double>(E) * kEdepScale);
  const long long m_fixed[3] = {__double2ll_rn(static_cast<double>(dir.x) * kEdepScale),
                                __double2ll_rn(static_cast<double>(dir.y) * kEdepScale),
                                __double2ll_rn(static_cast<double>(dir.z) * kEdepScale)};
  for (int i = 0; i < steps; ++i) {
    if (ix < 0 || ix >= nx || iy < 0 || iy >= ny || iz < 0 || iz >= nz) break;
    const size_t g = ix + static_cast<size_t>(iy) * nx + static_cast<size_t>(iz) * nx * ny;
    if (P.world_photon) atomicAdd(P.world_photon + g, 1);
    if (P.world_energy) atomicAdd(P.world_energy + g, static_cast<unsigned long long>(e_fixed));
    if (P.world_energy_squared) atomicAdd(P.world_energy_squared + g, static_cast<double>(E) * static_cast<double>(E));
    if (P.world_momentum)
      for (int a = 0; a < 3; ++a) atomicAdd(P.world_momentum + a * cells + g, static_cast<unsigned long long>(m_fixed[a]));
    p1 = add(p1, scale(increment, main_size));
    q = divv(sub(p1, lo), size);
    ix = __float2int_rz(q.x);
    iy = __float2int_rz(q.y);
    iz = __float2int_rz(q.z);
  }
}

// One point of the tracked slot's trajectory (gg_track_point).
__device__ __noinline__ void track_point(gg_track_point* points, int32_t* count, int capacity, int kind, int solid,
                                         int process, int history, V3 p, V3 d, float E) {
  const int i = atomicAdd(count, 1);
  if (i >= capacity) return;
  gg_track_point& t = points[i];
  t.kind = kind;
  t.solid = solid;
  t.process = process;
  t.history = history;
  t.E = E;
  t.position[0] = p.x;
  t.position[1] = p.y;
  t.position[2] = p.z;
  t.direction[0] = d.x;
  t.direction[1] = d.y;
  t.direction[2] = d.z;
  t.pad = 0.0f;
}

// Histogram of interaction sites in a CT detector module (the HISTOGRAM part of
// TrackThroughGGEMSSolidBox.cl:214-236), with the scatter histogram.
__device__ __noinline__ void box_histogram(const DevSolid& so, V3 p, bool scattered) {
  if (!so.histogram) return;
  V3 bmin = v3(so.border_min[0], so.border_min[1], so.border_min[2]);
  V3 es = divv(v3(so.box_size[0], so.box_size[1], so.box_size[2]),
               v3(static_cast<float>(so.virtual_element_number[0]), static_cast<float>(so.virtual_element_number[1]),
                  static_cast<float>(so.virtual_element_number[2])));
  V3 q = divv(sub(p, bmin), es);
  int ix = __float2int_rz(q.x), iy = __float2int_rz(q.y);
  if (ix >= 0 && iy >= 0 && ix < so.virtual_element_number[0] && iy < so.virtual_element_number[1]) {
    int idx = ix + iy * so.virtual_element_number[0];
    atomicAdd(so.histogram + idx, 1);
    if (so.scatter_histogram && scattered) atomicAdd(so.scatter_histogram + idx, 1);
  }
}

// ---- shared-memory staging with bounded waits ----
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Copies `bytes` (multiple of 16) from HBM into shared memory with
// cp.async.bulk and waits on an mbarrier for at most 2^22 polls (far longer
// than a 15 KB copy takes).  Returns false (and sets *error) when the copy did
// not complete in time; the CTA then exits, possibly with the copy still in
// flight, so the run reports GG_ERROR_TIMEOUT and the context must be
// recreated (include/ggems_b200.h).  Extra wait code here, even out of line,
// changes the register allocation of the whole kernel (more spills).
__device__ bool stage_tables(unsigned char* dst, const unsigned char* src, uint32_t bytes, uint64_t* bar, int* error) {
  constexpr uint32_t kChunk = 16384;
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
    for (uint32_t off = 0; off < bytes; off += kChunk) {
      uint32_t n = bytes - off < kChunk ? bytes - off : kChunk;
      asm volatile(
          "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
              smem_u32(dst + off)),
          "l"(src + off), "r"(n), "r"(smem_u32(bar))
          : "memory");
    }
  }
  uint32_t done = 0;
  for (int i = 0; i < (1 << 22) && !done; ++i) {
    asm volatile(
        "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0; selp.u32 %0, 1, 0, p; }"
        : "=r"(done)
        : "r"(smem_u32(bar))
        : "memory");
  }
  if (!done) atomicExch(error, 1);
  return __syncthreads_and(done) != 0;
}

extern __shared__ __align__(16) unsigned char g_smem[];

// Masks over a warp's stash records (one bit per record).
using StashMask = std::conditional_t<(kStashRecords > 32), unsigned long long, unsigned>;
__device__ __forceinline__ int stash_popc(unsigned m) { return __popc(m); }
__device__ __forceinline__ int stash_popc(unsigned long long m) { return __popcll(m); }
// 32-bit part h of a mask, and a 32-bit part placed at h
__device__ __forceinline__ unsigned stash_part(StashMask m, int h) {
  if constexpr (kStashRecords > 32) return static_cast<unsigned>(m >> (32 * h));
  else return m;
}
__device__ __forceinline__ StashMask stash_mask(unsigned part, int h) {
  if constexpr (kStashRecords > 32) return static_cast<StashMask>(part) << (32 * h);
  else return part;
}

// Register budget of a variant: what 256-thread blocks need to keep `blocks`
// of them resident per SM (64, 80 or 128 registers), fixed per kernel so that
// the block size stays a launch parameter (128, 256 or 512 threads).
constexpr int transport_registers(int blocks) { return (65536 / (kBlockThreads * blocks)) & ~7; }

// What bounds the kernel: the issue slots while photons cross large grids (CBCT
// 256^3: 69 % of them busy), and instruction fetches where events are frequent
// (36 projections through 64^3: 7.5 of the 14 cycles between two instructions of a
// warp), since the warps of an SM are in different parts of the code.  So the
// rare parts are kept short rather than fast: one copy of the exchange, of the
// exit from a solid and of the azimuth after an interaction, loops that are not
// unrolled, logarithms and exponentials out of line.  When the samplers and the
// sources went from 50 to 30 KB, CBCT of 1e8 went from 229 to 205 ms, 36
// projections from 32.8 to 28.8 and 64^3 dose from 2.25 to 2.09 ms (157 to 160, 26
// and 1.65 ms with the short voxel step).
//
// kFull: the scene has a meshed solid, a world grid or a tracked particle;
// kAux: the world walk and particle tracking are compiled in.  Scenes without
// them run variants compiled without that code, so its instructions and
// registers stay out of the voxel / detector (or mesh) hot loop.
// kDose: some solid tallies into a dose map.
// kBatch: several jobs (source runs) in one launch, each with its own solids.
// kStash: each warp keeps a second set of photons in shared memory and
// exchanges them with its lanes, so that lanes waiting for a rare phase track
// a parked photon meanwhile and rare rounds run on full warps.
// kAnyGrid: some voxel grid is refused by fast_steps (gg_runtime.cu), so the
// voxel steps take their general forms.  A variant of its own: the others' step
// keeps its registers.

template <bool kFull, bool kBatch, bool kDose, bool kAux, int kStash, bool kAnyGrid>
__global__ void __maxnreg__(transport_registers(kAux ? 2 : (kFull ? 3 : ((kBatch && kDose) || kStash == 2 ? 3 : 4))))
    transport_kernel(const __grid_constant__ TransportParams P) {
  // shared memory: [tables][solids][navigators][mbarrier][stash]
  unsigned char* tables = g_smem;
  DevSolid* scene_solids = reinterpret_cast<DevSolid*>(g_smem + (P.tables_in_smem ? P.table_bytes : 0));
  DevNavigator* navs = reinterpret_cast<DevNavigator*>(scene_solids + P.number_of_solids);
  uint64_t* bar = reinterpret_cast<uint64_t*>(navs + P.number_of_navigators);
  for (int i = threadIdx.x; i < P.number_of_solids; i += blockDim.x) scene_solids[i] = kBatch ? P.job_solids[i] : P.solids[i];
  for (int i = threadIdx.x; i < P.number_of_navigators; i += blockDim.x) navs[i] = P.navigators[i];
  Tab tab{P.table_blob, navs};
  if (P.tables_in_smem) {
    if (!stage_tables(tables, P.table_blob, P.table_bytes, bar, P.error)) return;
    tab.base = tables;
  } else {
    __syncthreads();
  }

  const size_t S = GG_MAXIMUM_PARTICLES;
  // Solids of the lane's current job: the shared-memory copy for a single
  // run, the job's own array (global memory) in a batched launch.  Where all
  // jobs have the same grids (the angles of a scan), the voxel steps read those
  // from the shared-memory copy of the first job's: lanes in different jobs then
  // read one address, not one each (36 projections of 1e6: 27.6 ms without, 26.3
  // with).
  const DevSolid* solids = scene_solids;
  int job = 0;
  const int number_of_jobs = kBatch ? P.number_of_jobs : 1;

  Kiss rng{0, 0, 0, 0, 0};
  Photon ph{};
  ph.solid_id = -1;
  uint32_t slot = ~0u;
  uint32_t histories_left = 0;
  int rounds = 0;
  int phase = kDone;
  int energy_id = 0;
  float cached_E = -1.0f;
  int cached_nav = -1;
  int pending = 0;  // process of a meshed solid's deferred interaction
  V3 inv_d = v3(0.0f, 0.0f, 0.0f);  // reciprocal(ph.d) while tracking inside a solid
  int history_number = -1;           // particle tracking: histories of the slot so far
  // particle tracking (full variant only): a point of this lane's photon when
  // its slot is the tracked one
  auto trk = [&](int kind, int solid, int process) {
    if (kAux && P.tracking_points && static_cast<int>(slot) == P.tracking_slot)
      track_point(P.tracking_points, P.tracking_count, P.tracking_capacity, kind, solid, process, history_number, ph.p,
                  ph.d, ph.E);
  };

  // A slot runs its histories of job 0, then of job 1, ... (each job is one
  // GGEMS source run; the slot's random stream carries over from run to run).
  // Returns false when the slot takes part in no job from `from` on.
  auto enter_job = [&](int from) -> bool {
#pragma unroll 1
    for (int j = from; j < number_of_jobs; ++j) {
      const DevJob& J = P.jobs[j];
      const uint32_t h = slot < J.q ? J.nb : (slot < J.q + 1 && J.r > 0 ? static_cast<uint32_t>(J.r) : 0u);
      if (h > 0) {
        if (kBatch) {
          job = j;
          solids = P.job_solids + static_cast<size_t>(j) * P.number_of_solids;
        }
        histories_left = h;
        ph.solid_id = -1;
        return true;
      }
    }
    return false;
  };
  // Grab the next slot: the lane takes slots_per_claim consecutive slots from
  // the work queue at a time and runs their photons one after another.  The
  // queue hands out runs starting at multiples of slots_per_claim (a power of
  // two), so the run is used up when the next slot is such a multiple (slot
  // starts at ~0u: the first call claims).
  auto next_slot = [&]() -> bool {
    if ((++slot & (P.slots_per_claim - 1)) == 0) slot = atomicAdd(P.slot_counter, P.slots_per_claim);
    if (slot >= P.number_of_slots) return false;
    rng = Kiss{P.rng[slot], P.rng[S + slot], P.rng[2 * S + slot], P.rng[3 * S + slot], P.rng[4 * S + slot]};
    return enter_job(0);
  };
  auto finish_slot = [&]() {
    P.rng[slot] = rng.s1;
    P.rng[S + slot] = rng.s2;
    P.rng[2 * S + slot] = rng.s3;
    P.rng[3 * S + slot] = rng.s4;
    P.rng[4 * S + slot] = rng.s5;
    if (P.particles.E) {
      P.particles.E[slot] = ph.E;
      P.particles.px[slot] = ph.p.x;
      P.particles.py[slot] = ph.p.y;
      P.particles.pz[slot] = ph.p.z;
      P.particles.dx[slot] = ph.d.x;
      P.particles.dy[slot] = ph.d.y;
      P.particles.dz[slot] = ph.d.z;
      P.particles.status[slot] = ph.status;
      P.particles.scatter[slot] = ph.scatter;
      P.particles.solid_id[slot] = ph.solid_id;
    }
  };

  auto end_history = [&]() {
    if (--histories_left > 0 || (kBatch && enter_job(job + 1))) {
      phase = kNewHistory;
    } else {
      finish_slot();
      phase = next_slot() ? kNewHistory : kDone;
    }
  };
  // End of track_through_*: back to the global frame; the history goes on
  // (FindSolid) unless the photon died.
  // why: 1 alive, 2 dead, 3 the history ends without a solid left.
  auto leave_solid = [&](const DevSolid* solid, int why) {
    const DevSolid& so = *solid;
    if (why == 3) {
    } else if (kFull && so.type == GG_SOLID_MESHED) {
      // A meshed solid tracks in world coordinates and, on leaving (dead or
      // not), carries the photon to its OBB boundary (TrackThroughGGEMSMeshSolid.cl:521-533).
      V3 mn = v3(so.border_min[0], so.border_min[1], so.border_min[2]);
      V3 mx = v3(so.border_max[0], so.border_max[1], so.border_max[2]);
      float dist = distance_to_aabb(g2l_pos(so.matrix, ph.p), g2l_dir(so.matrix, ph.d), mn, mx);
      float step = dist + kTolerance;
      ph.p = v3(ph.p.x + ph.d.x * step, ph.p.y + ph.d.y * step, ph.p.z + ph.d.z * step);
    } else {
      ph.p = l2g_pos(so.matrix, ph.p);
      ph.d = l2g_dir(so.matrix, ph.d);
    }
    if (why != 3) trk(why == 2 ? GG_TRACK_DEAD : GG_TRACK_LEAVE, -1, -1);
    if (why >= 2) end_history();
    else phase = kFind;
  };
  // A detector box takes whole steps in the rare rounds: nearly all of them end
  // in an interaction, and full warps sample those.  Against steps in the tracking
  // loop, 5e6 primaries on a panel without a phantom: water 300 mm 4.06 -> 2.51 ms,
  // 20 mm 2.35 -> 1.44, GOS 0.3 mm 1.09 -> 0.95, 10 mm at 140 keV 1.04 -> 0.97, but
  // 10 mm at 120 kVp, which stops all in one step, 0.87 -> 0.93; 46 curved modules
  // around a phantom, 2e7: 11.3 -> 9.0 ms.
  auto track_phase = [&](int type) {
    return type == GG_SOLID_VOXELIZED              ? kTrackVoxel
           : (kFull && type == GG_SOLID_MESHED) ? kTrackMesh
                                                : kInteract;
  };

  // BinarySearch of the photon's energy in navigator nav's bins, kept while both stay.
  auto find_energy = [&](int nav, int bins) {
    if (ph.E == cached_E && nav == cached_nav) return;
    energy_id = binary_search(ph.E, tab.energy_bins(nav), bins);
    cached_E = ph.E;
    cached_nav = nav;
  };
  auto find_tle_bin = [&](const DevSolid& so, int nav) -> int {
    return kDose && P.tle && so.dose_tle ? binary_search(ph.E, tab.attenuation(nav), GG_ATTENUATION_BINS) : 0;
  };
  // Moves the photon to the end of a step of length nid in a voxelized solid's
  // voxel or a detector box; whether that is inside the solid.
  // inner_min, inner_max: the solid's borders kTolerance inside (in_aabb's bounds).
  // tle_bin: tle_edep's e_index, where the solid's dose map uses it.
  auto step_to = [&](const DevSolid& so, bool voxel, int nav, int material, int tle_bin, float nid, int proc, V3 vmin,
                     V3 vmax, V3 inner_min, V3 inner_max) -> bool {
    if (kDose && P.photon_tracking && proc == GG_TRANSPORTATION && voxel && so.dose_map >= 0) {
      const DevDoseMap& dm = P.dose_maps[so.dose_map];
      if (dm.photon_tracking) {
        int id = dosel(dm, ph.p);
        if (id >= 0) atomicAdd(dm.photon_tracking + id, 1);
      }
    }
    ph.p = safety_outside(add(ph.p, scale(ph.d, nid)), vmin, vmax);
    const bool inside = !(ph.p.x < inner_min.x || ph.p.x > inner_max.x || ph.p.y < inner_min.y || ph.p.y > inner_max.y ||
                          ph.p.z < inner_min.z || ph.p.z > inner_max.z);
    if (kDose && P.tle && inside && voxel && so.dose_tle) {
      // The step's deposit depends only on the energy before the interaction,
      // so it is recorded here even when an interaction follows.
      dose_record(P.dose_maps[so.dose_map], tle_edep(tab.attenuation(nav), material, tle_bin, ph.E, nid), ph.p);
    }
    if (kAux && inside) trk(GG_TRACK_STEP, ph.solid_id, proc);
    return inside;
  };

  // ---- photon stash (kStash) ----
  // Per warp, kStashRecords photon records in shared memory (field f of record
  // r at w_stash[f * 32 + r]: a lane's accesses hit 32 different banks) and
  // three warp-uniform masks saying which records hold a photon ready to track
  // (st_ready), waiting for an interaction (st_int) or for a new history /
  // FindSolid round (st_find); a record in none of them is empty.  A photon
  // carries its whole state, slot and random stream included, so moving it
  // between a lane and a record never changes what its slot computes.
  constexpr int kWords = stash_words(kBatch, kAux);
  const int lane = threadIdx.x & 31;
  const unsigned lanes_below = (1u << lane) - 1u;
  uint32_t* w_stash = nullptr;
  int* w_index = nullptr;
  StashMask st_ready = 0, st_int = 0, st_find = 0;
  if (kStash) {
    uint32_t* base = reinterpret_cast<uint32_t*>(bar + 2);
    w_stash = base + (threadIdx.x >> 5) * (kWords * kStashRecords + kStashRecords);
    w_index = reinterpret_cast<int*>(w_stash + kWords * kStashRecords);
  }
  // Exchanges this lane's photon with record r.
  auto swap_record = [&](int r) {
    uint32_t* q = w_stash + r;
    auto xu = [&](int f, uint32_t& v) {
      const uint32_t t = q[f * kStashRecords];
      q[f * kStashRecords] = v;
      v = t;
    };
    auto xf = [&](int f, float& v) {
      const uint32_t t = q[f * kStashRecords];
      q[f * kStashRecords] = __float_as_uint(v);
      v = __uint_as_float(t);
    };
    auto xi = [&](int f, int& v) {
      const uint32_t t = q[f * kStashRecords];
      q[f * kStashRecords] = static_cast<uint32_t>(v);
      v = static_cast<int>(t);
    };
    xu(0, rng.s1);
    xu(1, rng.s2);
    xu(2, rng.s3);
    xu(3, rng.s4);
    xu(4, rng.s5);
    xf(5, ph.p.x);
    xf(6, ph.p.y);
    xf(7, ph.p.z);
    xf(8, ph.d.x);
    xf(9, ph.d.y);
    xf(10, ph.d.z);
    xf(11, ph.E);
    xf(12, ph.psd);
    xi(13, ph.solid_id);
    uint32_t packed = static_cast<uint32_t>(static_cast<uint8_t>(ph.status)) |
                      (static_cast<uint32_t>(static_cast<uint8_t>(ph.scatter)) << 8) |
                      (static_cast<uint32_t>(phase) << 16);
    xu(14, packed);
    ph.status = static_cast<int8_t>(packed & 0xffu);
    ph.scatter = static_cast<int8_t>((packed >> 8) & 0xffu);
    phase = static_cast<int>(packed >> 16);
    xu(15, slot);
    xu(16, histories_left);
    xi(17, rounds);
    xi(18, pending);
    xf(19, inv_d.x);
    xf(20, inv_d.y);
    xf(21, inv_d.z);
    xi(22, energy_id);
    xf(23, cached_E);
    xi(24, cached_nav);
    if (kBatch) {
      xi(25, job);
      solids = P.job_solids + static_cast<size_t>(job) * P.number_of_solids;
    }
    if (kAux) xi(kWords - 1, history_number);
  };
  // The k-th lane of `lanes` (in lane order) gets the k-th record of
  // `records`; -1 for the other lanes.  Called by the whole warp.
  auto match = [&](unsigned lanes, StashMask records) -> int {
    int ranked = 0;
#pragma unroll
    for (int h = 0; h < kStashRecords / 32; ++h) {
      const unsigned part = stash_part(records, h);
      if ((part >> lane) & 1u) w_index[ranked + __popc(part & lanes_below)] = lane + 32 * h;
      ranked += __popc(part);
    }
    __syncwarp();
    int r = -1;
    if ((lanes >> lane) & 1u) {
      const int k = __popc(lanes & lanes_below);
      if (k < ranked) r = w_index[k];
    }
    __syncwarp();
    return r;
  };
  auto is_rare = [](int ph_phase) { return ph_phase == kNewHistory || ph_phase == kFind || ph_phase == kInteract; };
  // Lanes of `lanes` exchange their photons with records of `records`; the
  // masks then say what each touched record holds.  Called by the whole warp.
  auto exchange = [&](unsigned lanes, StashMask records) {
    const int r = match(lanes, records);
    const int old = phase;
    if (r >= 0) swap_record(r);
    StashMask moved = 0, to_int = 0, to_find = 0, to_empty = 0;
#pragma unroll
    for (int h = 0; h < kStashRecords / 32; ++h) {
      const unsigned bit = (r >= 32 * h && r < 32 * h + 32) ? (1u << (r - 32 * h)) : 0u;
      moved |= stash_mask(__reduce_or_sync(0xffffffffu, bit), h);
      to_int |= stash_mask(__reduce_or_sync(0xffffffffu, old == kInteract ? bit : 0u), h);
      to_find |= stash_mask(__reduce_or_sync(0xffffffffu, (old == kNewHistory || old == kFind) ? bit : 0u), h);
      to_empty |= stash_mask(__reduce_or_sync(0xffffffffu, old == kDone ? bit : 0u), h);
    }
    st_int = (st_int & ~moved) | to_int;
    st_find = (st_find & ~moved) | to_find;
    st_ready = (st_ready & ~moved) | (moved & ~(to_int | to_find | to_empty));
  };

  if (kStash) {
    // Fill the records first: each lane claims a slot (a run of its own) for
    // records lane, lane + 32, ..., then one for itself.
#pragma unroll 1
    for (int h = 0; h < kStashRecords / 32; ++h) {
    phase = next_slot() ? kNewHistory : kDone;
    st_find |= stash_mask(__ballot_sync(0xffffffffu, phase == kNewHistory), h);
    swap_record(lane + 32 * h);  // the lane receives whatever the record held before: reset below
    slot = ~0u;
    histories_left = 0;
    rounds = 0;
    pending = 0;
    energy_id = 0;
    cached_E = -1.0f;
    cached_nav = -1;
    history_number = -1;
    ph = Photon{};
    ph.solid_id = -1;
    inv_d = v3(0.0f, 0.0f, 0.0f);
    if (kBatch) {
      job = 0;
      solids = scene_solids;
    }
    phase = kDone;
    }
  }
  if (next_slot()) phase = kNewHistory;

  // Warp-level phase scheduling.  Tracking steps (voxel or detector box) are
  // ~98 % of all steps; new histories, FindSolid/ProjectToSolid rounds and
  // Compton/Rayleigh sampling are rare but long.  Running every lane's phase
  // each iteration would execute the rare code for one or two lanes in most
  // iterations; instead the rare phases wait until regroup_lanes lanes need
  // them, or until they are at least regroup_ratio4/4 times as many as the
  // tracking lanes, and then run together.  A waiting lane draws no random
  // number and touches no tally, so waiting changes when it computes, never
  // what.
  const int regroup = P.regroup_lanes;
  const int ratio4 = P.regroup_ratio4;
  const int swap_lanes = P.stash_swap_lanes;
  const int round_photons = P.stash_round_photons;
  for (;;) {
    bool round = false, serve_interact = false;
    if (kStash) {
      // Two looks, with one copy of the exchange code for both.
      bool finished = false;
#pragma unroll 1
      for (int look = 0; look < 2; ++look) {
        const unsigned active = __ballot_sync(0xffffffffu, phase != kDone);
        const unsigned waiting = __ballot_sync(0xffffffffu, is_rare(phase));
        unsigned lanes = 0;
        StashMask records = 0;
        if (look == 0) {
          finished = active == 0 && (st_ready | st_int | st_find) == 0;
          if (finished) break;
          // Lanes waiting for a rare phase, and lanes without a photon, take
          // ready photons from the stash (once enough of them wait: an exchange
          // costs the warp two shared-memory accesses per word).
          lanes = waiting | ~active;
          if (__popc(lanes) >= min(swap_lanes, stash_popc(st_ready))) records = st_ready;
        } else {
          // A round of one kind of rare work when a full warp of it is waiting
          // (lanes and records), or when the waiting lanes are many against the
          // tracking ones and no ready photon is left to replace them.
          const unsigned w_int = __ballot_sync(0xffffffffu, phase == kInteract);
          const int n_int = __popc(w_int) + stash_popc(st_int);
          const int n_find = __popc(waiting & ~w_int) + stash_popc(st_find);
          const int n_wait = __popc(waiting), n_track = __popc(active & ~waiting);
          round = n_int + n_find > 0 &&
                  (n_int >= 32 || n_find >= 32 || n_int + n_find >= round_photons || n_track == 0 ||
                   (n_wait > 0 && (n_wait >= regroup || 4 * n_wait >= ratio4 * n_track)));
          if (round) {
            serve_interact = n_int >= 32 ? (n_find < 32 || n_int >= n_find) : (n_find < 32 && n_int >= n_find);
            // gather: lanes without a photon of the served kind take one from the stash
            lanes = ~(serve_interact ? w_int : (waiting & ~w_int));
            records = serve_interact ? st_int : st_find;
          }
        }
        if (records != 0 && lanes != 0) exchange(lanes, records);
      }
      if (finished) break;
    } else {
      const unsigned active = __ballot_sync(0xffffffffu, phase != kDone);
      if (active == 0) break;
      const unsigned tracking =
          __ballot_sync(0xffffffffu, phase == kTrackVoxel || (kFull && phase == kTrackMesh));
      const int n_other = __popc(active & ~tracking);
      round = n_other > 0 && (n_other >= regroup || 4 * n_other >= ratio4 * __popc(tracking));
      // A round serves one kind of rare work: the interaction samplers, or the
      // new-history / FindSolid chain, whichever more lanes wait for; the
      // others wait for the next round (their code paths stay out of this
      // one).  Measured +1.4 % on the CBCT projection.
      if (round) serve_interact = 2 * __popc(__ballot_sync(0xffffffffu, phase == kInteract)) >= n_other;
    }
    // A step or an interaction that ends the photon's stay in its solid sets
    // `leave` (1: alive, 2: dead; 3: no solid left) and `leaving`, and jumps to the one copy of
    // the exit code at the end of the loop body.
    int leave = 0;
    const DevSolid* leaving = nullptr;
    if (round) {
      if ((phase == kInteract) != serve_interact) continue;
      if (phase == kInteract) {
        const DevSolid& so = solids[ph.solid_id];
        const int nav = so.navigator;
        leaving = &so;
        int material = 0, proc = pending;
        if (!kFull || so.type != GG_SOLID_MESHED) {
          // A whole step through a voxelized solid
          // (track_through_ggems_voxelized_solid, TrackThroughGGEMSVoxelizedSolid.cl:133-310)
          // or a detector box (track_through_ggems_solid_box,
          // TrackThroughGGEMSSolidBox.cl:122-248): the same sampling and slab test
          // against the current voxel or the whole box (a grid of one voxel of
          // material 0), then each solid's own tail.
          const bool voxel = so.type == GG_SOLID_VOXELIZED;
          const int4 n0 = load4i(&navs[nav]);
          find_energy(nav, n0.x);
          const uint32_t pack = static_cast<uint32_t>(n0.y);
          const V3 bmin = v3(so.border_min[0], so.border_min[1], so.border_min[2]);
          const V3 bmax = v3(so.border_max[0], so.border_max[1], so.border_max[2]);
          const V3 vs = v3(so.voxel_sizes[0], so.voxel_sizes[1], so.voxel_sizes[2]);
          const int nx = so.number_of_voxels[0], ny = so.number_of_voxels[1], nz = so.number_of_voxels[2];
          V3 q = sub(ph.p, bmin);
          q = voxel ? divv(q, vs) : v3(0.0f, 0.0f, 0.0f);
          const int ix = __float2int_rz(q.x), iy = __float2int_rz(q.y), iz = __float2int_rz(q.z);
          if (ix >= nx || iy >= ny || iz >= nz || ix < 0 || iy < 0 || iz < 0) {
            ph.psd = kOutOfWorld;
            ph.solid_id = -1;
            leave = 1;
            goto exit_solid;
          }
          const V3 vmin = add(bmin, mul(v3(static_cast<float>(ix), static_cast<float>(iy), static_cast<float>(iz)), vs));
          const V3 vmax = voxel ? add(vmin, vs) : bmax;
          material = __ldg(so.labels + (ix + iy * nx + iz * nx * ny));
          const float4* row =
              reinterpret_cast<const float4*>(tab.base + static_cast<uint32_t>(n0.z)) +
              (material * n0.x + energy_id);
          const float cut = reinterpret_cast<const float*>(tab.base + static_cast<uint32_t>(n0.w))[material];
          float nid = next_interaction(draw_processes(rng, pack, P.three_processes != 0), pack, row[0], proc);
          ph.p = safety_inside(ph.p, vmin, vmax);
          const float dtb = distance_to_aabb(ph.p, ph.d, inv_d, vmin, vmax);
          if (dtb <= nid) {
            nid = dtb + kTolerance;
            proc = GG_TRANSPORTATION;
          }
          if (!step_to(so, voxel, nav, material, find_tle_bin(so, nav), nid, proc, vmin, vmax,
                       v3(so.inner_min[0], so.inner_min[1], so.inner_min[2]),
                       v3(so.inner_max[0], so.inner_max[1], so.inner_max[2]))) {
            ph.psd = kOutOfWorld;
            ph.solid_id = -1;
            leave = 1;
            goto exit_solid;
          }
          if (!voxel && ph.E < so.threshold) ph.status = GG_DEAD;
          if (proc != GG_COMPTON_SCATTERING && proc != GG_RAYLEIGH_SCATTERING) {
            if (!voxel) {
              if (proc == GG_PHOTOELECTRIC_EFFECT) {
                ph.status = GG_DEAD;
                ph.E = 0.0f;
                box_histogram(so, ph.p, ph.scatter == 1);
              }
            } else {
              if (proc == GG_PHOTOELECTRIC_EFFECT) {
                if (kDose && so.dose_map >= 0 && !so.dose_tle) dose_record(P.dose_maps[so.dose_map], ph.E, ph.p);
                ph.status = GG_DEAD;
                ph.E = 0.0f;
              }
              if (ph.E <= cut) {
                if (kDose && so.dose_map >= 0) dose_record(P.dose_maps[so.dose_map], ph.E, ph.p);
                ph.status = GG_DEAD;
              }
            }
            if (ph.status == GG_DEAD) {
              leave = 2;
              goto exit_solid;
            }
            phase = track_phase(so.type);
            goto resume;
          }
        }
        // The Compton / Rayleigh part of a tracking step (the tail of
        // track_through_*): sample the interaction, then tally as the step would.
        {
        float e0 = ph.E;
        scatter(ph, rng, proc, navs[nav], tab.energy_bins(nav), tab.sigma(nav), material, energy_id);
        trk(GG_TRACK_SCATTER, ph.solid_id, proc);
        if (so.type != GG_SOLID_BOX) {
          // voxelized and meshed solids flag scattering; boxes do not
          // (TrackThroughGGEMSVoxelizedSolid.cl:253, TrackThroughGGEMSMeshSolid.cl:484)
          ph.scatter = 1;
          if ((kDose && so.dose_map >= 0) && !so.dose_tle) dose_record(P.dose_maps[so.dose_map], e0 - ph.E, ph.p);
          if (ph.E <= tab.photon_cut(nav)[material]) {
            if ((kDose && so.dose_map >= 0)) dose_record(P.dose_maps[so.dose_map], ph.E, ph.p);
            ph.status = GG_DEAD;
          }
        } else if (proc == GG_COMPTON_SCATTERING) {
          box_histogram(so, ph.p, ph.scatter == 1);
        }
        if (ph.status == GG_DEAD) {
          leave = 2;
          goto exit_solid;
        }
        phase = track_phase(so.type);
        }
        goto resume;
      }
      if (phase == kNewHistory) {
        const DevSource& source = P.jobs[job].source;
        const PrimaryOut o = new_primary(rng, source);
        ph.p = o.p;
        ph.d = o.d;
        ph.E = o.E;
        rng = o.rng;
        ph.scatter = 0;
        ph.status = GG_ALIVE;
        ph.psd = kOutOfWorld;
        rounds = 0;
        phase = kFind;
        if (kAux) {
          ++history_number;
          trk(GG_TRACK_PRIMARY, -1, -1);
        }
      }
      if (phase != kFind) continue;
      bool end = rounds >= GG_MAX_LOOP;
      if (!end && P.number_of_solids == 0) {
        ++rounds;  // no navigator: the reference loop only counts iterations
      } else if (!end) {
        ++rounds;
        // particle_solid_distance_* (ParticleSolidDistanceGGEMS*.cl:43-108)
#pragma unroll 1
        for (int s = 0; s < P.number_of_solids; ++s) {
          if (ph.status == GG_DEAD || ph.psd == 0.0f) break;
          const DevSolid& so = solids[s];
          V3 mn = v3(so.border_min[0], so.border_min[1], so.border_min[2]);
          V3 mx = v3(so.border_max[0], so.border_max[1], so.border_max[2]);
          V3 lp = g2l_pos(so.matrix, ph.p);
          if (in_aabb(lp, mn, mx)) {
            ph.psd = 0.0f;
            ph.solid_id = s;
            break;
          }
          float dist = distance_to_aabb(lp, g2l_dir(so.matrix, ph.d), mn, mx);
          if (dist < ph.psd) {
            ph.psd = dist;
            ph.solid_id = s;
          }
        }
        if (kAux && P.world_dimensions[0] > 0 && ph.status != GG_DEAD) world_track(ph.p, ph.d, ph.E, ph.psd, P);
        // project_to_* (ProjectToGGEMS*.cl:44-129)
        if (ph.solid_id == -1) ph.status = GG_DEAD;
        if (ph.psd == kOutOfWorld) {
          ph.solid_id = -1;
          ph.status = GG_DEAD;
        } else if (ph.status != GG_DEAD) {
          const DevSolid& so = solids[ph.solid_id];
          ph.p = add(ph.p, scale(ph.d, ph.psd + kTolerance));
          V3 lp = g2l_pos(so.matrix, ph.p);
          lp = safety_inside(lp, v3(so.border_min[0], so.border_min[1], so.border_min[2]),
                             v3(so.border_max[0], so.border_max[1], so.border_max[2]));
          ph.p = l2g_pos(so.matrix, lp);
          ph.psd = 0.0f;
        }
        if (ph.status == GG_DEAD) {
          end = true;
          trk(GG_TRACK_DEAD, -1, -1);
        } else {
          // Enter the solid: switch to local coordinates (a meshed solid's
          // triangles are already in world coordinates).
          const DevSolid& so = solids[ph.solid_id];
          if (!kFull || so.type != GG_SOLID_MESHED) {
            ph.p = g2l_pos(so.matrix, ph.p);
            ph.d = g2l_dir(so.matrix, ph.d);
          }
          trk(GG_TRACK_ENTER, ph.solid_id, -1);
          phase = track_phase(so.type);
        }
      }
      if (end) {
        leave = 3;
        goto exit_solid;
      }
      if (phase == kFind) continue;
      goto resume;
    }
    if (phase != kTrackVoxel && !(kFull && phase == kTrackMesh)) continue;
    {

    // ---- tracking inside solid ph.solid_id ----
    // the solid's and navigator's per-step fields in six 16-byte loads
    // (DevSolid / DevNavigator lead with them)
    const DevSolid& so = solids[ph.solid_id];
    const DevSolid& grid = kBatch && P.shared_grids ? scene_solids[ph.solid_id] : so;
    const int4 s3 = load4i(&grid.number_of_voxels[0]);  // number_of_voxels xyz, navigator
    const int nav = s3.w;
    const int4 n0 = load4i(&navs[nav]);               // number_of_bins, process_pack, sigma / cut offsets
    const float4* sig = reinterpret_cast<const float4*>(tab.base + static_cast<uint32_t>(n0.z));
    find_energy(nav, n0.x);

    leaving = &so;
    const uint32_t pack = static_cast<uint32_t>(n0.y);
    if (!kFull || phase != kTrackMesh) {
      // Up to kTrackSteps steps through a voxelized solid that surely cross
      // their voxel, which 97 % do: no logarithm, no branch between the voxel
      // index and the step's end, so that the label's load, the three draws and
      // the slab test overlap.  Any other step is left undone, its random state
      // included, and taken as a whole in a round of the kInteract phase.  With a
      // logarithm and a division per process in every step CBCT of 1e8 primaries
      // took 270 ms, without 205 ms, and with the short forms below 172 ms.
      //
      // Every photon here is at least kTolerance inside the solid (the step's own
      // test of its end, or the one before the loop), and the host has checked
      // the grid for it (fast_steps in gg_runtime.cu).  That shortens three parts
      // of the step without a bit's difference:
      //  * a voxel index of such a position is in the grid;
      //  * the position is inside its voxel up to a few roundings, all of them
      //    below kTolerance, so safety_inside is a clamp;
      //  * from at least kTolerance inside the voxel every axis has one face
      //    behind and one ahead, so distance_to_aabb is the nearest face ahead.
      //    Its test that the ray stays 2 kTolerance in the box can only fail for
      //    a direction along x (else tmin is behind the photon, and two faces of
      //    different axes are 2 sqrt(2) kTolerance apart along any ray): steps
      //    shorter than that are left to the whole step.
      // The kAnyGrid variants keep the whole step's index, clamp and distance, for
      // any position in any grid, and spare the sampling as the others do: 2e6
      // primaries in 3 m of 10 mm voxels with dose 8.8 ms (21.7 as whole steps in the
      // rare rounds, 14.7 with a logarithm and a division per process in every
      // step), 5e6 in 5 um voxels 10.9 ms (20.6, 21.8).
      const float* cuts = reinterpret_cast<const float*>(tab.base + static_cast<uint32_t>(n0.w));
      const uint8_t* labels = so.labels;
      const int tle_bin = find_tle_bin(so, nav);
      if (!kAnyGrid) {
        const float4 c = load4f(&grid.inv_voxel_sizes[2]), d = load4f(&grid.inner_max[0]);
        if (!(ph.p.x >= c.y && ph.p.x <= d.x && ph.p.y >= c.z && ph.p.y <= d.y && ph.p.z >= c.w && ph.p.z <= d.z)) {
          phase = kInteract;
          continue;
        }
      }
#pragma unroll 1
      for (int k = 0; k < kTrackSteps; ++k) {
        const float4 a = load4f(&grid.border_min[0]);        // border_min xyz, voxel_sizes x
        const float4 b = load4f(&grid.voxel_sizes[1]);       // voxel_sizes yz, inv_voxel_sizes xy
        const float4 c = load4f(&grid.inv_voxel_sizes[2]);   // inv_voxel_sizes z, inner_min xyz
        const float4 d = load4f(&grid.inner_max[0]);         // inner_max xyz, label_bias
        const V3 bmin = v3(a.x, a.y, a.z), vs = v3(a.w, b.x, b.y);
        const V3 r = sub(ph.p, bmin);
        V3 i;  // the voxel, as floats
        uint32_t voxel;
        if (kAnyGrid) {
          const V3 q = divv(r, vs);
          const int ix = __float2int_rz(q.x), iy = __float2int_rz(q.y), iz = __float2int_rz(q.z);
          if (ix >= s3.x || iy >= s3.y || iz >= s3.z || ix < 0 || iy < 0 || iz < 0) {
            phase = kInteract;
            break;
          }
          i = v3(static_cast<float>(ix), static_cast<float>(iy), static_cast<float>(iz));
          voxel = static_cast<uint32_t>(ix + iy * s3.x + iz * s3.x * s3.y);
        } else {
          const V3 q = P.voxel_mode == kVoxelPow2 ? mul(r, v3(b.z, b.w, c.x))
                                                  : v3(quotient(r.x, vs.x, b.z), quotient(r.y, vs.y, b.w), quotient(r.z, vs.z, c.x));
          // trunc(q) without the conversion pipe: 2^23 + q rounded towards zero
          // holds trunc(q) in its low bits; label_bias takes the bits of the three
          // 2^23 out of the label's index
          const float mx = __fadd_rz(q.x, kTwo23), my = __fadd_rz(q.y, kTwo23), mz = __fadd_rz(q.z, kTwo23);
          voxel = (__float_as_uint(mz) * static_cast<uint32_t>(s3.y) + __float_as_uint(my)) * static_cast<uint32_t>(s3.x) +
                  __float_as_uint(mx) - __float_as_uint(d.w);
          i = v3(mx - kTwo23, my - kTwo23, mz - kTwo23);
        }
        const int material = __ldg(labels + voxel);
        const V3 vmin = add(bmin, mul(i, vs));
        const V3 vmax = add(vmin, vs);
        Kiss next = rng;
        const Draws draws = draw_processes(next, pack, P.three_processes != 0);
        V3 p;
        float dtb;
        bool whole = false;  // only the whole step is sure of the distance
        if (kAnyGrid) {
          p = safety_inside(ph.p, vmin, vmax);
          dtb = distance_to_aabb(p, ph.d, inv_d, vmin, vmax);
        } else {
          p = v3(fminf(fmaxf(ph.p.x, vmin.x + kTolerance), vmax.x - kTolerance),
                 fminf(fmaxf(ph.p.y, vmin.y + kTolerance), vmax.y - kTolerance),
                 fminf(fmaxf(ph.p.z, vmin.z + kTolerance), vmax.z - kTolerance));
          dtb = fminf(fminf(fmaxf((vmin.x - p.x) * inv_d.x, (vmax.x - p.x) * inv_d.x),
                            fmaxf((vmin.y - p.y) * inv_d.y, (vmax.y - p.y) * inv_d.y)),
                      fmaxf((vmin.z - p.z) * inv_d.z, (vmax.z - p.z) * inv_d.z));
          whole = dtb < 2.0f * kTolerance;
        }
        const float4 sigma = sig[material * n0.x + energy_id];
        if (!(surely_crosses(draws, sigma, dtb) && !whole && ph.E > cuts[material])) {
          phase = kInteract;
          break;
        }
        rng = next;
        ph.p = p;
        if (!step_to(so, true, nav, material, tle_bin, dtb + kTolerance, GG_TRANSPORTATION, vmin, vmax, v3(c.y, c.z, c.w),
                     v3(d.x, d.y, d.z))) {
          ph.psd = kOutOfWorld;
          ph.solid_id = -1;
          leave = 1;
          break;
        }
      }
    }
    else if (kFull && phase == kTrackMesh) do {
      // track_through_ggems_meshed_solid, TrackThroughGGEMSMeshSolid.cl:385-518:
      // the parity of the crossing count says whether the photon is inside the
      // mesh; outside, it jumps to the first crossing.  Material 0.
      const MeshCrossings x =
          mesh_crossings(ph.p, ph.d, inv_d, so.mesh_nodes, so.mesh_node_count, so.mesh_triangles, so.mesh_bvh);
      if (x.count == 0) {
        ph.psd = kOutOfWorld;
        ph.solid_id = -1;
        leave = 1;
        break;
      }
      V3 next = x.first;
      if ((x.count & 1) == 0) {
        ph.p = x.first;
        next = x.second;
      }
      int proc;
      float nid = next_interaction(draw_processes(rng, pack, P.three_processes != 0), pack,
                                   sig[energy_id], proc);
      const float dx = next.x - ph.p.x, dy = next.y - ph.p.y, dz = next.z - ph.p.z;
      const float to_next = sqrtf(dx * dx + dy * dy + dz * dz);
      if (to_next <= nid) {
        nid = to_next + kTolerance;
        proc = GG_TRANSPORTATION;
        if ((kDose && so.dose_map >= 0)) {
          const DevDoseMap& dm = P.dose_maps[so.dose_map];
          if (dm.photon_tracking) {
            int id = dosel(dm, ph.p);
            if (id >= 0) atomicAdd(dm.photon_tracking + id, 1);
          }
        }
      }
      ph.p = add(ph.p, scale(ph.d, nid));
      trk(GG_TRACK_STEP, ph.solid_id, proc);
      if (proc == GG_COMPTON_SCATTERING || proc == GG_RAYLEIGH_SCATTERING) {
        pending = proc;
        phase = kInteract;
        continue;
      }
      if (proc == GG_PHOTOELECTRIC_EFFECT) {
        if ((kDose && so.dose_map >= 0)) dose_record(P.dose_maps[so.dose_map], ph.E, ph.p);
        ph.status = GG_DEAD;
        ph.E = 0.0f;
      }
      if (ph.E <= reinterpret_cast<const float*>(tab.base + static_cast<uint32_t>(n0.w))[0]) {
        if ((kDose && so.dose_map >= 0)) dose_record(P.dose_maps[so.dose_map], ph.E, ph.p);
        ph.status = GG_DEAD;
      }
      if (ph.status == GG_DEAD) leave = 2;
    } while (0);
    }
  exit_solid:
    if (leave) leave_solid(leaving, leave);
    continue;
  resume:
    inv_d = reciprocal(ph.d);
  }
}

// compute_dose_ggems_{voxelized,meshed}_solid, ComputeDoseGGEMSVoxelizedSolid.cl:53-121,
// ComputeDoseGGEMSMeshSolid.cl:53-114
__global__ void compute_dose_kernel(DoseParams P) {
  const DevDoseMap& dm = P.map;
  int id = blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= dm.total_number_of_dosels) return;
  int z = id / dm.slice_number_of_dosels;
  int x = (id - z * dm.slice_number_of_dosels) % dm.number_of_dosels[0];
  int y = (id - z * dm.slice_number_of_dosels) / dm.number_of_dosels[0];
  float px = static_cast<float>(x) * dm.size_of_dosels[0] +
             static_cast<float>(dm.number_of_dosels[0] - 1) * (-0.5f * dm.size_of_dosels[0]);
  float py = static_cast<float>(y) * dm.size_of_dosels[1] +
             static_cast<float>(dm.number_of_dosels[1] - 1) * (-0.5f * dm.size_of_dosels[1]);
  float pz = static_cast<float>(z) * dm.size_of_dosels[2] +
             static_cast<float>(dm.number_of_dosels[2] - 1) * (-0.5f * dm.size_of_dosels[2]);
  int material = 0;  // meshed solids (ComputeDoseGGEMSMeshSolid.cl:90): material 0, no labels
  if (P.labels) {
    int vx = __float2int_rz((px - P.border_min[0]) / P.voxel_sizes[0]);
    int vy = __float2int_rz((py - P.border_min[1]) / P.voxel_sizes[1]);
    int vz = __float2int_rz((pz - P.border_min[2]) / P.voxel_sizes[2]);
    material = P.labels[vx + vy * P.number_of_voxels[0] + vz * P.number_of_voxels[0] * P.number_of_voxels[1]];
  }
  float vol = dm.size_of_dosels[0] * dm.size_of_dosels[1] * dm.size_of_dosels[2];
  constexpr float kGCm3 = 6.241509704e+21f / 1.e3f;  // g/cm3
  constexpr float kGy = 1.0e-12f;
  float density = P.is_water_reference ? 1.0f * kGCm3 : P.density[material];
  double edep = static_cast<double>(static_cast<long long>(dm.edep[id])) / kEdepScale;
  P.dose[id] = density < P.minimum_density
                   ? 0.0f
                   : static_cast<float>(static_cast<double>(P.scale_factor) * edep / static_cast<double>(density) /
                                        static_cast<double>(vol) / static_cast<double>(kGy));
  if (P.uncertainty) {
    int hit = dm.hit ? dm.hit[id] : 0;
    if (hit > 1 && edep != 0.0) {
      double e2 = dm.edep_squared ? dm.edep_squared[id] : 0.0;
      double sum2 = edep * edep;
      P.uncertainty[id] = static_cast<float>(sqrt((hit * e2 - sum2) / ((hit - 1) * sum2)));
    } else {
      P.uncertainty[id] = 1.0f;
    }
  }
}

}  // namespace

namespace {
using TransportKernel = void (*)(TransportParams);
// kFull: meshed solids, world grid or particle tracking (dose code always in),
// kAux: world grid or particle tracking; otherwise the dose-map code is
// compiled in only for scenes that tally dose.
// kStash: the photon stash (voxel / detector scenes without world grid or
// particle tracking).
// kAnyGrid: as TransportParams::voxel_mode says.
template <bool kAnyGrid>
TransportKernel transport_variant(bool mesh, bool batch, bool dose, bool aux, int stash) {
  constexpr bool A = kAnyGrid;
  if (aux) return batch ? transport_kernel<true, true, true, true, 0, A> : transport_kernel<true, false, true, true, 0, A>;
  if (mesh) {
    if (stash) return batch ? transport_kernel<true, true, true, false, 2, A> : transport_kernel<true, false, true, false, 2, A>;
    return batch ? transport_kernel<true, true, true, false, 0, A> : transport_kernel<true, false, true, false, 0, A>;
  }
  if (stash == 1) {
    if (dose) return batch ? transport_kernel<false, true, true, false, 1, A> : transport_kernel<false, false, true, false, 1, A>;
    return batch ? transport_kernel<false, true, false, false, 1, A> : transport_kernel<false, false, false, false, 1, A>;
  }
  if (stash == 2) {
    if (dose) return batch ? transport_kernel<false, true, true, false, 2, A> : transport_kernel<false, false, true, false, 2, A>;
    return batch ? transport_kernel<false, true, false, false, 2, A> : transport_kernel<false, false, false, false, 2, A>;
  }
  if (dose) return batch ? transport_kernel<false, true, true, false, 0, A> : transport_kernel<false, false, true, false, 0, A>;
  return batch ? transport_kernel<false, true, false, false, 0, A> : transport_kernel<false, false, false, false, 0, A>;
}
TransportKernel transport_variant(const TransportParams& p, bool mesh, bool dose, bool aux, int stash) {
  const bool batch = p.number_of_jobs > 1;
  return p.voxel_mode == kVoxelGeneral ? transport_variant<true>(mesh, batch, dose, aux, stash)
                                       : transport_variant<false>(mesh, batch, dose, aux, stash);
}
}  // namespace

void launch_transport(const TransportParams& p, int grid, int threads, size_t smem, void* stream, bool mesh, bool dose,
                      bool aux, int stash) {
  transport_variant(p, mesh, dose, aux, stash)<<<grid, threads, smem, static_cast<cudaStream_t>(stream)>>>(p);
}

namespace {

// Siddon-style ray march (Amanatides-Woo voxel walk) from the source to the
// centre of detector element (i, j), in the phantom's frame: sum of
// mu[label] x chord length.  Element centres follow the detector histogram's
// binning (element (i, j) covers [bmin + i es, bmin + (i+1) es) in x, y).
//
// One launch walks every projection of a call (blockIdx.z), a block 32 x 8
// elements, a warp 8 x 4 of them (neighbouring rays read the same label lines).
// The walk's position does not depend on the labels, so kRayBatch steps are
// taken at a time: their labels load together, then the chords are summed in
// order.  What bounds it is the walk's instructions (~100 steps a ray); the
// label volume stays in L2.  360 projections of 256^2 rays through 64^3 labels:
// 12.0 ms as one launch each (one dependent label load a step, few rays in
// flight), 2.9 ms now; 8 projections of 333^2 1.32x.
constexpr int kRayBatch = 4;
constexpr int kRayThreads = 256;
__global__ void __launch_bounds__(kRayThreads) line_integral_kernel(const __grid_constant__ ProjectorParams P) {
  __shared__ float mu[257];  // by label; 256: a step past the ray's end
  for (int k = threadIdx.x; k < 257; k += kRayThreads) mu[k] = k < P.number_of_materials && k < 256 ? P.mu[k] : 0.0f;
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = blockIdx.x * 32 + (warp & 3) * 8 + (lane & 7), j = blockIdx.y * 8 + (warp >> 2) * 4 + (lane >> 3);
  if (i >= P.elements[0] || j >= P.elements[1]) return;
  for (int proj = blockIdx.z; proj < P.count; proj += gridDim.z) {
    const RayFrame& R = P.frames[proj];
    const V3 local_pixel = v3(R.detector_min[0] + (static_cast<float>(i) + 0.5f) * R.element_size[0],
                              R.detector_min[1] + (static_cast<float>(j) + 0.5f) * R.element_size[1], 0.0f);
    const V3 pixel = l2g_pos(R.detector_matrix, local_pixel);
    const V3 s = g2l_pos(P.phantom_matrix, v3(R.source[0], R.source[1], R.source[2]));
    const V3 e = g2l_pos(P.phantom_matrix, pixel);
    const float dv[3] = {e.x - s.x, e.y - s.y, e.z - s.z};
    const float sv[3] = {s.x, s.y, s.z};
    float t0 = 0.0f, t1 = 1.0f;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      if (fabsf(dv[a]) < 1e-12f) {
        if (sv[a] < P.border_min[a] || sv[a] > P.border_max[a]) t1 = -1.0f;
      } else {
        float ta = (P.border_min[a] - sv[a]) / dv[a], tb = (P.border_max[a] - sv[a]) / dv[a];
        if (ta > tb) {
          float t = ta;
          ta = tb;
          tb = t;
        }
        t0 = fmaxf(t0, ta);
        t1 = fminf(t1, tb);
      }
    }
    float sum = 0.0f;
    if (t1 > t0) {
      const float length = sqrtf(dv[0] * dv[0] + dv[1] * dv[1] + dv[2] * dv[2]);
      int left[3], stride[3];  // voxels ahead on the axis; label offset of a step
      float tmax[3], tdelta[3];
      const float tm = 0.5f * (t0 + t1);
      int offset = 0;
      int pitch = 1;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        // start voxel: the one containing the entry point (nudged inside)
        const float pa = sv[a] + fminf(t0 + 1e-6f * (t1 - t0), tm) * dv[a];
        int k = static_cast<int>(floorf((pa - P.border_min[a]) / P.voxel_sizes[a]));
        k = min(max(k, 0), P.number_of_voxels[a] - 1);
        offset += k * pitch;
        if (dv[a] > 0.0f) {
          left[a] = P.number_of_voxels[a] - 1 - k;
          stride[a] = pitch;
          tmax[a] = (P.border_min[a] + (k + 1) * P.voxel_sizes[a] - sv[a]) / dv[a];
          tdelta[a] = P.voxel_sizes[a] / dv[a];
        } else if (dv[a] < 0.0f) {
          left[a] = k;
          stride[a] = -pitch;
          tmax[a] = (P.border_min[a] + k * P.voxel_sizes[a] - sv[a]) / dv[a];
          tdelta[a] = -P.voxel_sizes[a] / dv[a];
        } else {
          left[a] = 0x7fffffff;
          stride[a] = 0;
          tmax[a] = FLT_MAX;
          tdelta[a] = FLT_MAX;
        }
        pitch *= P.number_of_voxels[a];
      }
      float t = t0;
      bool on = true;
      int guard = 4 * (P.number_of_voxels[0] + P.number_of_voxels[1] + P.number_of_voxels[2]);
      while (on) {
        int label[kRayBatch];
        float chord[kRayBatch];
#pragma unroll
        for (int k = 0; k < kRayBatch; ++k) {
          const bool x_first = tmax[0] < tmax[1];
          const bool z_next = !((x_first ? tmax[0] : tmax[1]) < tmax[2]);
          const bool ax = x_first && !z_next, ay = !x_first && !z_next;
          const float tn = fminf(z_next ? tmax[2] : (ax ? tmax[0] : tmax[1]), t1);
          label[k] = on ? static_cast<int>(__ldg(P.labels + offset)) : 256;
          chord[k] = tn - t;
          t = tn;
          const int ahead = z_next ? left[2] : (ax ? left[0] : left[1]);
          on = on && !(t >= t1) && ahead > 0 && --guard > 0;
          offset += on ? (z_next ? stride[2] : (ax ? stride[0] : stride[1])) : 0;
          left[0] -= ax ? 1 : 0;
          left[1] -= ay ? 1 : 0;
          left[2] -= z_next ? 1 : 0;
          tmax[0] = ax ? tmax[0] + tdelta[0] : tmax[0];
          tmax[1] = ay ? tmax[1] + tdelta[1] : tmax[1];
          tmax[2] = z_next ? tmax[2] + tdelta[2] : tmax[2];
        }
#pragma unroll
        for (int k = 0; k < kRayBatch; ++k) {
          const float add = mu[label[k]] * chord[k] * length;
          sum = label[k] < 256 ? sum + add : sum;
        }
      }
    }
    const size_t o = (static_cast<size_t>(proj) * P.elements[1] + j) * P.elements[0] + i;
    if (P.network_input) {
      P.out[2 * o] = expf(-sum);
      P.out[2 * o + 1] = sum;
    } else {
      P.out[o] = sum;
    }
  }
}

}  // namespace

void launch_line_integrals(const ProjectorParams& p, void* stream) {
  dim3 grid((p.elements[0] + 31) / 32, (p.elements[1] + 7) / 8, p.count < 65535 ? p.count : 65535);
  line_integral_kernel<<<grid, kRayThreads, 0, static_cast<cudaStream_t>(stream)>>>(p);
}

void launch_compute_dose(const DoseParams& p, void* stream) {
  int n = p.map.total_number_of_dosels;
  compute_dose_kernel<<<(n + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(p);
}

cudaError_t configure_transport(const TransportParams& p, size_t smem, int threads, int* blocks_per_sm, bool mesh,
                                bool dose, bool aux, int stash) {
  auto kernel = transport_variant(p, mesh, dose, aux, stash);
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (e != cudaSuccess) return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, kernel, threads, smem);
}

cudaError_t set_rayleigh_fit(const float* pp /* 9*101 */) {
  return cudaMemcpyToSymbol(c_rayleigh_pp, pp, sizeof(float) * 9 * 101);
}

}  // namespace gg
