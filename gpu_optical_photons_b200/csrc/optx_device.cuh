// optx_device.cuh - device physics of the optx engine (sm_100a).
//
// One photon step of next-event transport in an axis-aligned box, with the
// physics of the reference's include/optphot/transport.hpp:55-145 and the
// random-number layout of include/optphot/philox.hpp:97-149 (paths relative to
// the reference project zmeskma/GPU_Optical_photons). The arithmetic of every
// quantity follows the reference expression for expression, so that a build
// without FMA contraction and with the portable math of pmath.hpp (OPTX_EXACT=1)
// reproduces the reference CPU histories bit for bit; the fast build
// (OPTX_EXACT=0) calls CUDA's logf / sincosf / cbrtf and lets nvcc contract.
//
// What is restructured for the GPU (values unchanged):
//  * Random words come from a two-block window (8 words of the photon's Philox
//    stream, blocks b and b+1). A step reads its 2..5 words at offsets o..o+4
//    of the window with register selects, and the only Philox call site is
//    after the step, when block b has been used up. The reference instead
//    tests for an empty buffer at every draw, so a warp runs Philox once per
//    draw site at which any lane has run dry.
//  * The three outcomes share one move (pos + d * dir) and the two rotations
//    (Rayleigh scatter, Lambertian bounce) and the two Fresnel interfaces
//    (readout, polished) share one code path each, which keeps lanes with
//    different outcomes on the same instructions.
//  * Reflection on an axis-aligned face is the sign flip of one component and
//    cos_i = |dir[axis]|: both are what reflect() / dot() of fresnel.hpp and
//    transport.hpp:105-106 produce bit for bit for a unit axis normal.
//  * Parameters derived from SimParams once on the host (inv_speed, (n1/n2)^2)
//    are computed with the same float operations as the reference.
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#ifndef OPTX_EXACT
#define OPTX_EXACT 0
#endif
#ifndef OPTX_APPROX  // 1: compiled with --use_fast_math
#define OPTX_APPROX 0
#endif

namespace optx {

// ---------------------------------------------------------------------------
// Parameters as the kernels see them (built by the host from optx_params and
// optx_faces, see capi.cu: make_dev_params). 112 bytes in 16-byte groups of what is
// read together, so that a record in memory costs a step two 128-bit loads, a
// polished face two 64-bit loads and a Philox block one (load_step, step_act): with
// one 32-bit load per field the batch ran 19 of them per warp step and took 9.08 ms
// against 8.9.
struct __align__(16) DevParams {
  float hx, hy, hz, inv_speed;             // inv_speed = n_scint / c  (transport.hpp:74)
  float abs_length, scat_length;
  uint32_t max_steps;
  uint32_t surf_bits;                      // 2 bits per face 0..4: Polished/Black/Specular/Lambertian
  float n_det, eta2_det, n_out, eta2_out;  // eta2 = (n_scint / n)^2 (fresnel.hpp:32-33)
  float n_scint, tau;
  uint32_t key_lo, key_hi;
  float refl0, refl1, refl2, refl3;        // reflectivity of faces 0..4
  float refl4;
  uint32_t flags;                          // kOrdinary
  float inv2hx, inv2hy;                    // 1 / (2 hx), 1 / (2 hy) rounded to nearest (xy_bin)
  float src_x, src_y, src_z;
  uint32_t source;                         // 0 point, 1 uniform in the volume, 2 genstep segment
};
static_assert(sizeof(DevParams) == 112, "DevParams layout");
// The wide and the indexed reads of a record in memory rely on these places.
static_assert(offsetof(DevParams, abs_length) == 16 && offsetof(DevParams, surf_bits) == 28 &&
                  offsetof(DevParams, n_det) == 32 && offsetof(DevParams, n_out) == 40 &&
                  offsetof(DevParams, key_lo) % 8 == 0 &&
                  offsetof(DevParams, key_hi) == offsetof(DevParams, key_lo) + 4 &&
                  offsetof(DevParams, refl4) == offsetof(DevParams, refl0) + 16,
              "DevParams layout");

// Device-side structure-of-arrays photon records (29 bytes per photon).
struct DevRecords {
  uint8_t* fate;
  uint32_t* n_boundary;
  uint32_t* n_scatter;
  float *t, *x, *y, *z, *path;
};

// DevParams::flags. kOrdinary: sizes, indices and source lie where the branch-free
// quotients below are exact (ordinary_params in capi.cu); a run with any other
// record takes the IEEE divisions.
enum : uint32_t { kOrdinary = 1u };

enum : uint32_t { kPolished = 0, kBlack = 1, kSpecular = 2, kLambertian = 3 };
enum : uint32_t { kDetected = 0, kAbsorbedBulk = 1, kAbsorbedSurface = 2, kEscaped = 3, kMaxSteps = 4 };
constexpr int kReadoutFace = 5;
constexpr float kInf = __builtin_huge_valf();

// ---------------------------------------------------------------------------
// Philox4x32-10 (Salmon et al., SC11), counter {block, 0, id_lo, id_hi},
// key {seed_lo, seed_hi} (philox.hpp:64-76, :86-115). The 32x32->64 products
// map to one wide multiply each; the key schedule is warp-uniform when all
// lanes share a seed.
__device__ __forceinline__ uint4 philox10(uint4 c, uint32_t k0, uint32_t k1) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const unsigned long long p0 = static_cast<unsigned long long>(0xD2511F53u) * c.x;
    const unsigned long long p1 = static_cast<unsigned long long>(0xCD9E8D57u) * c.z;
    c = make_uint4(static_cast<uint32_t>(p1 >> 32) ^ c.y ^ k0, static_cast<uint32_t>(p1),
                   static_cast<uint32_t>(p0 >> 32) ^ c.w ^ k1, static_cast<uint32_t>(p0));
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  return c;
}

// The same with the round keys of one key made beforehand (philox_keys), in the
// constant bank: no key additions for the batched kernels, whose photons usually
// share a key, and for the history kernel (tally of 1e8 bar photons 43.2 -> 42.0 ms,
// 10 registers fewer).
struct PhiloxKeys {
  uint32_t k0[10], k1[10];
};
__device__ __forceinline__ uint4 philox10(uint4 c, const PhiloxKeys& K) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const unsigned long long p0 = static_cast<unsigned long long>(0xD2511F53u) * c.x;
    const unsigned long long p1 = static_cast<unsigned long long>(0xCD9E8D57u) * c.z;
    c = make_uint4(static_cast<uint32_t>(p1 >> 32) ^ c.y ^ K.k0[r], static_cast<uint32_t>(p1),
                   static_cast<uint32_t>(p0 >> 32) ^ c.w ^ K.k1[r], static_cast<uint32_t>(p0));
  }
  return c;
}
__device__ __forceinline__ uint4 philox10(uint4 c, uint2 key) { return philox10(c, key.x, key.y); }
__device__ __forceinline__ uint4 philox_counter(uint32_t block, uint64_t id) {
  return make_uint4(block, 0u, static_cast<uint32_t>(id), static_cast<uint32_t>(id >> 32));
}

// (bits >> 8) + 1 times 2^-24, in (0, 1], exact (philox.hpp:82-84).
__device__ __forceinline__ float to_uniform(uint32_t bits) {
  // One FMA for the addition and the scaling: the sum is at most 2^24, so exact.
  return fmaf(__uint2float_rn(bits >> 8), 1.0f / 16777216.0f, 1.0f / 16777216.0f);
}

// The photon's random stream as a window of two consecutive Philox blocks.
// Invariant between steps: w[0..3] = block `blk`, w[4..7] = block `blk + 1`,
// next unread word at w[o], o in [0, 3]; so a step can read 5 words.
// draws() = 4 * blk + o is the reference's PhiloxStream::draws().
// The photon id and key are not stored: callers pass them (the key lives in the
// parameters, the id is first id + photon index), which keeps the per-lane state
// at 10 registers.
struct Rng {
  uint32_t w[8];
  uint32_t o, blk;

  // Starts (draws = 0) or resumes the stream of photon `id` after `draws` words
  // (philox.hpp:117-134): blocks draws/4 and draws/4 + 1 fill the window, as two
  // independent Philox chains (instruction-level parallelism: -1 % on the batch,
  // -3 % on the history kernel).
  template <class K>
  __device__ __forceinline__ void init(uint64_t id, const K& key, uint32_t draws) {
    const uint32_t block = draws >> 2;
    set(philox10(philox_counter(block, id), key), philox10(philox_counter(block + 1u, id), key), draws);
  }
  // The window from its two blocks, `draws` words into the stream.
  __device__ __forceinline__ void set(const uint4& b0, const uint4& b1, uint32_t draws) {
    w[0] = b0.x; w[1] = b0.y; w[2] = b0.z; w[3] = b0.w;
    w[4] = b1.x; w[5] = b1.y; w[6] = b1.z; w[7] = b1.w;
    blk = draws >> 2;
    o = draws & 3u;
  }
  __device__ __forceinline__ uint32_t draws() const { return 4u * blk + o; }

  // Word o + I of the window, I a compile-time index in [0, 4]: three selects.
  template <int I>
  __device__ __forceinline__ uint32_t word() const {
    const uint32_t lo = (o & 1u) ? w[I + 1] : w[I];
    const uint32_t hi = (o & 1u) ? w[I + 3] : w[I + 2];
    return (o & 2u) ? hi : lo;
  }
  template <int I>
  __device__ __forceinline__ float uniform() const { return to_uniform(word<I>()); }

  // Consumes k words; slides the window (one Philox call per block used up).
  template <class K>
  __device__ __forceinline__ void advance(uint32_t k, uint64_t id, const K& key) {
    o += k;
#pragma unroll 1
    while (o >= 4u) slide(philox10(philox_counter(blk + 2u, id), key));
  }
  // The same when block blk + 2 has been made already.
  template <class K>
  __device__ __forceinline__ void advance(uint32_t k, uint64_t id, const K& key, const uint4& next) {
    o += k;
    if (o >= 4u) slide(next);
    if (o >= 4u) slide(philox10(philox_counter(blk + 2u, id), key));
  }
  // Moves the window on by one block; b: block blk + 2.
  __device__ __forceinline__ void slide(const uint4& b) {
    w[0] = w[4]; w[1] = w[5]; w[2] = w[6]; w[3] = w[7];
    w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
    ++blk;
    o -= 4u;
  }
};

// The photon's random stream as up to 12 unread uniforms (three Philox blocks) in a
// ring in shared memory, for kernels that refill all lanes of a warp together: a
// photon holds three registers of it instead of ten, a step reads its words with
// indexed loads instead of selects, words are turned into uniforms once, and with
// more than a step's words in hand most warp steps need one Philox pass, not two (a
// photon starts with 9 words or 10, a bounce reads 5). For the batched variants,
// whose registers are the scarcest: against the register window the 4096-event batch
// ran 8.61 -> 8.13 ms, 512 events of gensteps 0.854 -> 0.807. One configuration keeps
// the register window: a polished or specular step reads three words, and the ring's
// shared-memory round trip cost more (polished cube 1e8 photons 8.48 -> 9.26 ms, bar
// 26.8 -> 28.1, Lambertian cube 14.13 -> 14.10), except in the adjoint replays.
// Invariant between steps: av >= 5; rp + av is a multiple of 4, so a block is one
// aligned 128-bit store.
constexpr uint32_t kWindowWords = 12u;
struct Window {
  float* ring;    // this photon's kWindowWords places
  uint32_t rp;    // place of the next unread word
  uint32_t av;    // unread words
  uint32_t made;  // Philox blocks made so far
  __device__ __forceinline__ uint32_t draws() const { return 4u * made - av; }
  // j mod kWindowWords for j < 2 kWindowWords: the difference wraps around below 0.
  static __device__ __forceinline__ uint32_t wrap(uint32_t j) { return min(j, j - kWindowWords); }
  template <int I>
  __device__ __forceinline__ float uniform() const { return ring[wrap(rp + I)]; }
  __device__ __forceinline__ void consume(uint32_t k) {
    rp = wrap(rp + k);
    av -= k;
  }
  // Appends block `made`; av <= kWindowWords - 4.
  __device__ __forceinline__ void put(const uint4& v) {
    *reinterpret_cast<float4*>(ring + wrap(rp + av)) =
        make_float4(to_uniform(v.x), to_uniform(v.y), to_uniform(v.z), to_uniform(v.w));
    av += 4u;
    ++made;
  }
};
// The stream of one of a warp's last photons: a ring of kLoneWords uniforms in shared
// memory that the whole warp fills (wave_kernel, drain), word w at place w mod kLoneWords.
constexpr uint32_t kLoneWords = 64u;
struct LoneStream {
  const float* ring;
  uint32_t next;  // words used so far (the reference's PhiloxStream::draws())
  template <int I>
  __device__ __forceinline__ float uniform() const { return ring[(next + I) & (kLoneWords - 1u)]; }
};

// Words a step reads at most, and room for another block.
constexpr uint32_t kStepWords = 5u, kWindowRoom = kWindowWords - 4u;

// ---------------------------------------------------------------------------
// Correctly rounded quotient, reciprocal and square root without a branch: the
// hardware's approximation, refined with FMA residuals (Markstein, IBM J. Res.
// Dev. 34(1), 1990: with y the rounded reciprocal and q within an ulp of a / b,
// q + (a - b q) y rounds to the quotient; the square root likewise from
// g = x / sqrt(x) and its residual x - g^2). They equal the IEEE operations on the
// ranges the step uses them on; tests/cuda/ieee_check.cu compares them with
// __fdiv_rn, __frcp_rn and __fsqrt_rn. nvcc's own operators guard every range with a
// check and a branch to a slow path: a step has about a dozen of them, one after
// another, and the branches also keep the chains from overlapping. Measured against
// the operators (1e7 photons, kernel time): Lambertian cube 1.90 -> 1.64 ms, polished
// cube 1.36 -> 1.22 ms; 4096-event batch 9.81 -> 9.27 ms. The APPROX build keeps
// the operators: --use_fast_math already turns them into the approximations.
#if OPTX_APPROX
__device__ __forceinline__ float m_rcp(float b) { return 1.0f / b; }
__device__ __forceinline__ float m_div(float a, float b) { return a / b; }
__device__ __forceinline__ float m_sqrt(float x) { return sqrtf(x); }
#else
__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rsqrt_approx(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float lg2_approx(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// 1 / b for 2^-100 <= |b| <= 2^100; NaN for b = 0.
__device__ __forceinline__ float m_rcp(float b) {
  const float y = rcp_approx(b);
  return fmaf(y, fmaf(-b, y, 1.0f), y);
}
// a / b for b as above and a = 0 or |a| >= 2^-100, when the quotient is normal (or
// 0); NaN for b = 0.
__device__ __forceinline__ float m_div(float a, float b) {
  const float y = m_rcp(b);
  const float q = a * y;
  return fmaf(fmaf(-b, q, a), y, q);
}
// sqrt(x) for x = 0 or 2^-60 <= x <= 2^60.
__device__ __forceinline__ float m_sqrt(float x) {
  const float y = rsqrt_approx(fmaxf(x, 0x1p-60f));  // finite at 0, where g = 0 x y = 0
  const float g = x * y;
  return fmaf(fmaf(-g, g, x), 0.5f * y, g);
}
#endif

// ---------------------------------------------------------------------------
// Math policy (pmath.hpp:134-158). Fast: CUDA's library functions. Exact: the
// portable functions built from correctly rounded operations only (the
// reference's pmath.hpp:62-130 methods: atanh series for log, exact quarter-turn
// reduction and Taylor polynomials for sin/cos, Newton iterations for cbrt),
// compiled without FMA contraction.
#if OPTX_EXACT
__device__ __forceinline__ float m_log(float x) {
  const uint32_t bits = __float_as_uint(x);
  int e = static_cast<int>((bits >> 23) & 0xffu) - 127;
  float m = __uint_as_float((bits & 0x007fffffu) | 0x3f800000u);
  if (m > 1.41421356f) {
    m = 0.5f * m;
    ++e;
  }
  const float s = m_div(m - 1.0f, m + 1.0f);
  const float s2 = s * s;
  const float poly = 1.0f + s2 * (1.0f / 3.0f + s2 * (1.0f / 5.0f + s2 * (1.0f / 7.0f +
                     s2 * (1.0f / 9.0f + s2 * (1.0f / 11.0f)))));
  const float fe = static_cast<float>(e);
  return fe * 6.9313812256e-01f + (2.0f * s * poly + fe * 9.0580006145e-06f);
}
__device__ __forceinline__ void m_sincos_turns(float u, float& s, float& c) {
  const float v = 4.0f * u;
  float q = floorf(v);
  float r = v - q;
  if (r > 0.5f) {
    r -= 1.0f;
    q += 1.0f;
  }
  const float x = r * 1.57079632679489662f;
  const float x2 = x * x;
  const float sp = x * (1.0f + x2 * (-1.0f / 6.0f + x2 * (1.0f / 120.0f +
                   x2 * (-1.0f / 5040.0f + x2 * (1.0f / 362880.0f)))));
  const float cp = 1.0f + x2 * (-0.5f + x2 * (1.0f / 24.0f + x2 * (-1.0f / 720.0f +
                   x2 * (1.0f / 40320.0f + x2 * (-1.0f / 3628800.0f)))));
  const int quadrant = static_cast<int>(q) & 3;
  const float ss = (quadrant & 1) ? cp : sp;
  const float cc = (quadrant & 1) ? sp : cp;
  s = (quadrant & 2) ? -ss : ss;
  c = ((quadrant + 1) & 2) ? -cc : cc;
}
__device__ __forceinline__ float m_cbrt(float x) {
  float y = __uint_as_float(__float_as_uint(x) / 3u + 0x2a514067u);
#pragma unroll
  for (int i = 0; i < 4; ++i) y = y - m_div(y * y * y - x, 3.0f * y * y);
  return y;
}
#else
__device__ __forceinline__ float m_log(float x) { return logf(x); }
__device__ __forceinline__ void m_sincos_turns(float u, float& s, float& c) {
  const float a = 6.28318530717958647692f * u;
#if !OPTX_APPROX
  // u is in (0, 1]: without this the reduction of huge arguments is compiled in,
  // with a 28-byte local array (measured: -2.6 % on the Lambertian cube).
  __builtin_assume(fabsf(a) <= 7.0f);
#endif
  sincosf(a, &s, &c);
}
__device__ __forceinline__ float m_cbrt(float x) { return cbrtf(x); }
#endif

// ---------------------------------------------------------------------------
struct Photon {
  float px, py, pz, dx, dy, dz, t, path;
  uint32_t nb, ns;
};

// Per-photon counters needed by the adjoint's score terms.
struct ScoreAux {
  uint32_t n_refl;  // reflections at painted (specular / Lambertian) faces
  float t_emit;     // sampled emission time
};

// GP: P is a record in global memory, read with wide or indexed loads; a kernel
// parameter is read field by field and with selects instead (indexing it would copy
// the parameters to local memory). Records do not change while a kernel that steps
// photons runs.
template <bool GP>
__device__ __forceinline__ float face_refl(const DevParams& P, int face) {
  if (GP) return __ldg(&P.refl0 + face);
  float r = P.refl0;
  r = (face == 1) ? P.refl1 : r;
  r = (face == 2) ? P.refl2 : r;
  r = (face == 3) ? P.refl3 : r;
  r = (face == 4) ? P.refl4 : r;
  return r;
}

// The parameters that every step reads.
struct StepParams {
  float hx, hy, hz, inv_speed, abs_length, scat_length;
  uint32_t max_steps, surf_bits;
};
template <bool GP>
__device__ __forceinline__ StepParams load_step(const DevParams& P) {
  if (GP) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(&P)), b = __ldg(reinterpret_cast<const float4*>(&P) + 1);
    return {a.x, a.y, a.z, a.w, b.x, b.y, __float_as_uint(b.z), __float_as_uint(b.w)};
  }
  return {P.hx, P.hy, P.hz, P.inv_speed, P.abs_length, P.scat_length, P.max_steps, P.surf_bits};
}

// Branch-free orthonormal basis (Duff et al., JCGT 6(1) 2017) and rotation
// about `axis` by polar cosine ct and azimuth 2 pi * phi_u (vec3.hpp:35-53).
__device__ __forceinline__ void rotate_about(float ax, float ay, float az, float ct, float phi_u,
                                             float& ox, float& oy, float& oz) {
  const float sign = copysignf(1.0f, az);
  const float a = -m_rcp(sign + az);
  const float b = ax * ay * a;
  const float t1x = 1.0f + sign * ax * ax * a, t1y = sign * b, t1z = -sign * ax;
  const float t2x = b, t2y = sign + ay * ay * a, t2z = -ay;
  const float st = m_sqrt(fmaxf(0.0f, 1.0f - ct * ct));
  float sp, cp;
  m_sincos_turns(phi_u, sp, cp);
  const float A = st * cp, B = st * sp;
  const float x = A * t1x + B * t2x + ct * ax;
  const float y = A * t1y + B * t2y + ct * ay;
  const float z = A * t1z + B * t2z + ct * az;
  const float inv = m_rcp(m_sqrt(x * x + y * y + z * z));
  ox = inv * x;
  oy = inv * y;
  oz = inv * z;
}

// Rayleigh polar cosine by Cardano inversion of F(mu) = (mu^3 + 3 mu + 4) / 8
// (sampling.hpp:39-44).
__device__ __forceinline__ float rayleigh_cos(float u) {
  const float q = 4.0f * u - 2.0f;
  const float s = m_sqrt(q * q + 1.0f);
  // One cube-root call site: cbrt(q + s) for q >= 0, 1 / cbrt(s - q) otherwise.
  const bool pos = q >= 0.0f;
  const float c = m_cbrt(pos ? q + s : s - q);
  const float a = pos ? c : m_rcp(c);
  return fminf(1.0f, fmaxf(-1.0f, a - m_rcp(a)));
}

// Unpolarised Fresnel reflectance from n1 into n2 (fresnel.hpp:30-46);
// eta2 = (n1 / n2)^2 precomputed with the same float operations.
__device__ __forceinline__ float fresnel_R(float n1, float n2, float eta2, float cos_i) {
  if (n1 == n2) return 0.0f;
#if OPTX_EXACT || OPTX_APPROX
  const float sin2_t = eta2 * fmaxf(0.0f, 1.0f - cos_i * cos_i);
#else
  const float sin2_t = __fmul_rn(eta2, fmaxf(0.0f, fmaf(-cos_i, cos_i, 1.0f)));
#endif
  if (sin2_t >= 1.0f) return 1.0f;
  const float cos_t = sqrtf(1.0f - sin2_t);
#if OPTX_EXACT || OPTX_APPROX
  const float rs = (n1 * cos_i - n2 * cos_t) / (n1 * cos_i + n2 * cos_t);
  const float rp = (n2 * cos_i - n1 * cos_t) / (n2 * cos_i + n1 * cos_t);
  return 0.5f * (rs * rs + rp * rp);
#else
  // nvcc's contraction of these expressions, spelled out: left to the compiler it
  // would depend on what the caller computes beside them.
  const float rs = fmaf(n1, cos_i, __fmul_rn(-n2, cos_t)) / fmaf(n1, cos_i, __fmul_rn(n2, cos_t));
  const float rp = fmaf(n2, cos_i, __fmul_rn(-n1, cos_t)) / fmaf(n2, cos_i, __fmul_rn(n1, cos_t));
  return 0.5f * fmaf(rs, rs, __fmul_rn(rp, rp));
#endif
}

// u <= fresnel_R(...): the step needs only this outcome, never R itself, so the
// comparison is made on approximate values, multiplied out (no division), and
// fresnel_R decides where they leave it open. With p = n1 c + n2 ct and
// q = n2 c + n1 ct, R = (v^2 + w^2) / (2 (p q)^2), v = (n1 c - n2 ct) q,
// w = (n2 c - n1 ct) p. Both sides are off by less than 2^-17 (p q)^2 (the
// approximate square root by 2^-22 of itself; fresnel_R's own rounding
// included), a quarter of the margin; within 2^-10 of total internal
// reflection, where sqrt(1 - sin2_t) magnifies the rounding of sin2_t, and outside
// the ordinary range, fresnel_R decides too. Measured against calling it always:
// batch 9.27 -> 9.09 ms, gradient run of 1e6 photons 0.272 -> 0.259 ms. Without
// `asked` the outcome is not used and may be left open.
__device__ __forceinline__ bool fresnel_reflects(float n1, float n2, float eta2, float cos_i, float u,
                                                 uint32_t flags, bool asked = true) {
#if OPTX_APPROX
  (void)flags, (void)asked;
  return u <= fresnel_R(n1, n2, eta2, cos_i);
#else
  const float c2 = 1.0f - eta2 * fmaxf(0.0f, 1.0f - cos_i * cos_i);
  const float ct = c2 * rsqrt_approx(fmaxf(c2, 0x1p-60f));
  const float a = n1 * cos_i, b = n2 * ct, c = n2 * cos_i, d = n1 * ct;
  const float p = a + b, q = c + d, pq = p * q, v = (a - b) * q, w = (c - d) * p;
  const float den = pq * pq;
  const float diff = fmaf(v, v, w * w) - 2.0f * u * den;
  bool r = c2 < 0.0f || diff > 0.0f;
  const bool open = !(fabsf(diff) > 0x1p-15f * den) && !(c2 <= -0x1p-10f);
  if (asked && (open || fabsf(c2) < 0x1p-10f || !(flags & kOrdinary))) r = u <= fresnel_R(n1, n2, eta2, cos_i);
  return r;
#endif
}

// Emission (transport.hpp:55-67): position (3 draws, volume source only),
// isotropic direction (2), exponential emission time (1).
//
// Genstep segments (source 2, an extension with no reference counterpart): the
// photon starts at src + u1 (end - src) on the segment from src to end and at
// time t0 + u2 dt + the exponential decay time; u3 is drawn and unused, so the
// photon consumes the same six words as the reference's sources. `seg` holds
// (end x, y, z, t0) and (dt, -, -, -) of the photon's genstep (null otherwise).
constexpr uint32_t kSourceSegment = 2u;

// `u`: the first six uniforms of the stream. Returns the words used (3 or 6).
template <bool AUX>
__device__ __forceinline__ uint32_t start_photon(const DevParams& P, Photon& s, const float (&u)[6], ScoreAux& aux,
                                                 const float4* seg = nullptr) {
  float t_start = 0.0f, ua = u[0], ub = u[1], ue = u[2];
  if (P.source == 0u) {
    s.px = P.src_x;
    s.py = P.src_y;
    s.pz = P.src_z;
  } else {
    if (P.source == 1u) {
      s.px = P.hx * (2.0f * u[0] - 1.0f);
      s.py = P.hy * (2.0f * u[1] - 1.0f);
      s.pz = P.hz * (2.0f * u[2] - 1.0f);
    } else {
      const float4 e = seg[0], w = seg[1];
      s.px = P.src_x + u[0] * (e.x - P.src_x);
      s.py = P.src_y + u[0] * (e.y - P.src_y);
      s.pz = P.src_z + u[0] * (e.z - P.src_z);
      t_start = e.w + u[1] * w.x;
    }
    ua = u[3];
    ub = u[4];
    ue = u[5];
  }
  const float ct = 2.0f * ua - 1.0f;
  const float st = m_sqrt(fmaxf(0.0f, 1.0f - ct * ct));
  float sp, cp;
  m_sincos_turns(ub, sp, cp);
  s.dx = st * cp;
  s.dy = st * sp;
  s.dz = ct;
  s.t = P.tau > 0.0f ? -P.tau * m_log(ue) : 0.0f;
  if (AUX) aux.t_emit = s.t;
  if (P.source == kSourceSegment) s.t = t_start + s.t;
  s.path = 0.0f;
  s.nb = 0u;
  s.ns = 0u;
  return P.source == 0u ? 3u : 6u;
}
// The same with the register window, from the start of the stream.
template <class K>
__device__ __forceinline__ void start_photon(const DevParams& P, const K& key, Photon& s, Rng& r, uint64_t id,
                                             ScoreAux& aux) {
  r.init(id, key, 0u);
  const float u[6] = {to_uniform(r.w[0]), to_uniform(r.w[1]), to_uniform(r.w[2]),
                      to_uniform(r.w[3]), to_uniform(r.w[4]), to_uniform(r.w[5])};
  r.advance(start_photon<false>(P, s, u, aux), id, key);
}

// How a step is laid out. kBranches: the Fresnel decision and the painted faces behind
// branches, the rare IEEE box exit behind one after the quotients, which then stand in
// one block with what precedes them (Lambertian and polished cube, bar 1e8 photons
// -0.5 to -1 %). kFlat: every lane computes both and selects, for batches, where some
// lane of a warp nearly always needs each (4096 events 8.10 -> 7.87 ms, with the
// reordered box exit; in one configuration's main loop the bar gains a percent without
// it). kLone: as kBranches but with the box exit's branch first, for the last photons
// of a warp (bar 3e4 photons 209 us, 222 with the branch after).
enum StepShape { kBranches, kFlat, kLone };

// A step's interaction, decided by step_move: absorption, a scatter, or a hit on the
// face across the x, y or z axis on the side that `along`, the direction component
// across it, points to. Predicates rather than a face number: the step asks for the
// axis a dozen times (62 integer comparisons per warp step of the batch with one).
struct Hit {
  bool absorb, scatter, x, y, z;
  float along;
  __device__ __forceinline__ bool surface() const { return !absorb && !scatter; }
  __device__ __forceinline__ bool pos() const { return along > 0.0f; }
  __device__ __forceinline__ bool readout() const { return z && pos(); }
  __device__ __forceinline__ int face() const { return (x ? 0 : (y ? 2 : 4)) + (pos() ? 1 : 0); }
  // A surface hit or scatter as a number, 0..5 or kHitScatter, and back with the
  // photon's direction.
  static constexpr int kHitScatter = 6;
  __device__ __forceinline__ int code() const { return scatter ? kHitScatter : face(); }
  static __device__ __forceinline__ Hit of(int code, const Photon& s) {
    const bool x = code < 2, y = code == 2 || code == 3;
    return {false, code == kHitScatter, x, y, code == 4 || code == 5, x ? s.dx : (y ? s.dy : s.dz)};
  }
};
static_assert(kReadoutFace == 5, "the +z face");

// Distance to the box exit: per axis only the face the photon moves towards
// (geometry.hpp:25-46), an axis it does not move along being skipped.
__device__ __forceinline__ float box_exit_ieee(const StepParams& P, const Photon& s, Hit& hit) {
  float dist = kInf;
  hit.x = hit.y = hit.z = false;
  hit.along = fabsf(s.dz);  // no face (a position that is not a number): clamped, polished
  {
    const float tt = ((s.dx > 0.0f ? P.hx : -P.hx) - s.px) / s.dx;
    if (s.dx != 0.0f && tt < dist) { dist = tt; hit.x = true; hit.along = s.dx; }
  }
  {
    const float tt = ((s.dy > 0.0f ? P.hy : -P.hy) - s.py) / s.dy;
    if (s.dy != 0.0f && tt < dist) { dist = tt; hit.x = false; hit.y = true; hit.along = s.dy; }
  }
  {
    const float tt = ((s.dz > 0.0f ? P.hz : -P.hz) - s.pz) / s.dz;
    if (s.dz != 0.0f && tt < dist) { dist = tt; hit.x = hit.y = false; hit.z = true; hit.along = s.dz; }
  }
  return dist;
}

// The same for ordinary records, where m_div is exact: the quotient of an axis the
// photon does not move along is NaN and fminf passes over it; an earlier axis wins
// a tie, as in the order of the comparisons above. (A direction component is 0 or
// far above 2^-100: it comes out of sums of products of uniforms and sines.)
template <StepShape SHAPE = kBranches>
__device__ __forceinline__ float box_exit(const StepParams& P, uint32_t flags, const Photon& s, Hit& hit) {
#if OPTX_APPROX
  return box_exit_ieee(P, s, hit);
#else
  if (SHAPE == kLone && !(flags & kOrdinary)) return box_exit_ieee(P, s, hit);
  const float tx = m_div(copysignf(P.hx, s.dx) - s.px, s.dx);
  const float ty = m_div(copysignf(P.hy, s.dy) - s.py, s.dy);
  const float tz = m_div(copysignf(P.hz, s.dz) - s.pz, s.dz);
  float dist = fminf(fminf(tx, ty), tz);
  hit.x = tx == dist;
  hit.y = !hit.x && ty == dist;
  hit.z = !hit.x && !hit.y;
  hit.along = hit.x ? s.dx : (hit.y ? s.dy : s.dz);
  if (SHAPE != kLone && !(flags & kOrdinary)) dist = box_exit_ieee(P, s, hit);
  return dist;
#endif
}

#if !OPTX_APPROX
// Bounds of -log(u): lo <= -m_log(u) <= hi for every uniform u (all 2^24 checked in
// tests/cuda/ieee_check.cu), from the hardware's base-2 logarithm. Products with a
// length keep the order, rounding being monotonic.
__device__ __forceinline__ float log_lo(float lg2) { return fmaf(lg2, -0.69314718f * (1.0f - 0x1p-18f), -0x1p-20f); }
__device__ __forceinline__ float log_hi(float lg2) { return fmaf(lg2, -0.69314718f * (1.0f + 0x1p-18f), 0x1p-20f); }
#endif

// First half of a step (transport.hpp:71-97): the exponential absorption and
// scattering distances (window words 0 and 1), the box exit, and the move to the
// nearest of the three. Returns the interaction; the window is not advanced.
// PATH: the path length is kept; ENDS: the final state of every photon is recorded,
// so the position of an absorption counts (tallies and replays do not use it).
// Which of the three comes first is decided on the bounds of the two distances; the
// logarithms themselves are taken only where a photon moves by one of them, or where
// the bounds leave it open (~1e-5 of the steps). Kernel times against taking both
// always, with a face number in place of Hit's predicates: polished cube 1e8 photons
// 8.11 -> 7.70 ms, bar 25.9 -> 25.1, Lambertian cube 13.6 -> 13.1, batch 8.08 -> 7.87.
template <bool PATH = true, bool ENDS = true, StepShape SHAPE = kBranches, class R>
__device__ __forceinline__ Hit step_move(const StepParams& P, uint32_t flags, Photon& s, const R& r) {
  const float u_abs = r.template uniform<0>(), u_sca = r.template uniform<1>();
  Hit hit;
  const float dist = fmaxf(box_exit<SHAPE>(P, flags, s, hit), 0.0f);
  float d = dist;
#if OPTX_APPROX
  {
#else
  const float ga = lg2_approx(u_abs), gs = lg2_approx(u_sca);
  const float a_lo = P.abs_length * log_lo(ga), s_lo = P.scat_length * log_lo(gs);
  const float a_hi = P.abs_length * log_hi(ga), s_hi = P.scat_length * log_hi(gs);
  hit.absorb = a_hi < dist && a_hi < s_lo;
  hit.scatter = s_hi < dist && s_hi < a_lo;
  if (ENDS && hit.absorb) d = -P.abs_length * m_log(u_abs);
  if (hit.scatter) {
    d = -P.scat_length * m_log(u_sca);
  } else if (!hit.absorb && !(a_lo >= dist && s_lo >= dist)) {
#endif
    const float s_abs = (P.abs_length == kInf) ? kInf : -P.abs_length * m_log(u_abs);
    const float s_sca = (P.scat_length == kInf) ? kInf : -P.scat_length * m_log(u_sca);
    hit.absorb = s_abs < dist && s_abs <= s_sca;
    hit.scatter = !hit.absorb && s_sca < dist;
    d = hit.absorb ? s_abs : (hit.scatter ? s_sca : dist);
  }
  float nx = s.px + d * s.dx, ny = s.py + d * s.dy, nz = s.pz + d * s.dz;
  if (hit.surface()) {  // snap onto the face plane, clamp in-plane (geometry.hpp:57-63)
    nx = hit.x ? copysignf(P.hx, s.dx) : fminf(fmaxf(nx, -P.hx), P.hx);
    ny = hit.y ? copysignf(P.hy, s.dy) : fminf(fmaxf(ny, -P.hy), P.hy);
    nz = hit.z ? copysignf(P.hz, s.dz) : fminf(fmaxf(nz, -P.hz), P.hz);
  }
  s.px = nx;
  s.py = ny;
  s.pz = nz;
  s.t = s.t + d * P.inv_speed;
  if (PATH) s.path = s.path + d;
  return hit;
}

// Surface model of the face that was hit (the readout face is always polished).
__device__ __forceinline__ uint32_t face_model(uint32_t surf_bits, const Hit& hit) {
  return hit.readout() ? kPolished : ((surf_bits >> (2 * hit.face())) & 3u);
}

// Second half of a step (transport.hpp:98-145): the interaction `hit` at the
// photon's position. Returns true while the photon is alive, with the words of the
// window that the step used in `used` (the caller advances the window); otherwise
// `fate` is set and the photon sits at its final interaction.
// The outcome of every interaction comes first, as a few predicates (kept,
// scattered, mirrored, diffuse), then one pass each of the rotation and the mirror
// flip for all lanes that need it: fewer branches than a body per outcome (per warp
// step of the batch 47 of them, not 66; Lambertian cube 1e7 photons 1.63 -> 1.55 ms).
template <bool AUX, bool GP = false, StepShape SHAPE = kBranches, class R>
__device__ __forceinline__ bool step_act(const DevParams& P, uint32_t surf_bits, uint32_t flags, Photon& s, const R& r,
                                         uint32_t& fate, ScoreAux& aux, const Hit& hit, uint32_t& used) {
  // The window's words 2..4 as uniforms, once for every outcome (measured -2 % on
  // the batch against drawing them where an outcome uses them).
  const float u2 = r.template uniform<2>(), u3 = r.template uniform<3>(), u4 = r.template uniform<4>();
  const bool scattered = hit.scatter, surface = hit.surface();
  const uint32_t model = face_model(surf_bits, hit);
  // Readout face: interface to n_det, transmitted = detected; other polished faces:
  // interface to n_out, transmitted = escaped (transport.hpp:108-128).
  auto reflects = [&](bool asked) {
    float2 n2;  // index beyond the face, eta2
    if (GP) n2 = __ldg(reinterpret_cast<const float2*>(&P.n_det) + (hit.readout() ? 0 : 1));
    else n2 = hit.readout() ? make_float2(P.n_det, P.eta2_det) : make_float2(P.n_out, P.eta2_out);
    return fresnel_reflects(GP ? __ldg(&P.n_scint) : P.n_scint, n2.x, n2.y, fabsf(hit.along), u2, flags, asked);
  };
  // Painted reflector: absorbed with 1 - R; black: always (transport.hpp:129-144).
  bool kept = false;
  if constexpr (SHAPE == kFlat && !OPTX_APPROX) {
    const bool polished = surface && model == kPolished;
    const bool reflected = reflects(polished);
    const float refl = face_refl<GP>(P, hit.face());
    const bool kept_paint = surface & (model != kBlack) & (u2 <= refl);
    kept = polished ? reflected : kept_paint;
    fate = polished ? (hit.readout() ? kDetected : kEscaped) : (surface ? kAbsorbedSurface : kAbsorbedBulk);
    if (AUX) aux.n_refl += (kept_paint && !polished) ? 1u : 0u;
    if (surface) ++s.nb;
  } else if (surface) {
    if (model == kPolished) {
      kept = reflects(true);
      fate = hit.readout() ? kDetected : kEscaped;
    } else {
      kept = model != kBlack && u2 <= face_refl<GP>(P, hit.face());
      fate = kAbsorbedSurface;
      if (AUX && kept) ++aux.n_refl;
    }
    ++s.nb;
  } else {
    fate = kAbsorbedBulk;
  }
  if (scattered) ++s.ns;
  const bool diffuse = kept && model == kLambertian, mirrored = kept && !diffuse;
  const bool live = kept || scattered;
  if (diffuse || scattered) {
    float ax = s.dx, ay = s.dy, az = s.dz, ct, phi_u = u3;
    if (scattered) {
      ct = rayleigh_cos(u2);
    } else {
      // Lambertian about the inward normal -n (signed zeros as in -face_normal()).
      const float sg = hit.pos() ? -1.0f : 1.0f;
      ax = hit.x ? sg : -0.0f;
      ay = hit.y ? sg : -0.0f;
      az = hit.z ? sg : -0.0f;
      ct = m_sqrt(u3);
      phi_u = u4;
    }
    rotate_about(ax, ay, az, ct, phi_u, s.dx, s.dy, s.dz);
  }
  if (mirrored && hit.x) s.dx = -s.dx;
  if (mirrored && hit.y) s.dy = -s.dy;
  if (mirrored && hit.z) s.dz = -s.dz;
  if (live) fate = kMaxSteps;
  used = scattered ? 4u : (diffuse ? 5u : 3u);
  return live;
}

// One step (transport.hpp:71-145): move, then interact. `flags`: those that hold for
// every record of the run. False when the photon has ended, with its fate, or has
// made max_steps steps (the fate is then kMaxSteps); true with the words used.
template <bool AUX, bool GP = false, bool PATH = true, StepShape SHAPE = kBranches, class R>
__device__ __forceinline__ bool step_photon(const DevParams& P, uint32_t flags, Photon& s, const R& r, uint32_t& fate,
                                            ScoreAux& aux, uint32_t& used) {
  const StepParams q = load_step<GP>(P);
  const Hit hit = step_move<PATH, PATH && !AUX, SHAPE>(q, flags, s, r);
  const bool live = step_act<AUX, GP, SHAPE>(P, q.surf_bits, flags, s, r, fate, aux, hit, used);
  return live && s.nb + s.ns < q.max_steps;
}

// Tally binning (transport.hpp:170-181); tscale = time_bins / time_max in float.
__device__ __forceinline__ uint32_t time_bin(float t, float tscale, uint32_t time_bins) {
  const float f = t * tscale;
  return (f >= static_cast<float>(time_bins)) ? time_bins : static_cast<uint32_t>(f);
}
// a / b for 0 <= a <= b from y = 1 / b rounded to nearest: the product and two
// FMA corrections. With y the correctly rounded reciprocal and q1 within an ulp
// of a / b, q1 + (a - b q1) y rounds to the correctly rounded quotient
// (Markstein, IBM J. Res. Dev. 34(1), 1990), so this equals the IEEE division
// a / b whenever a / b does not underflow; checked on B200 against __fdiv_rn
// for every a in [b 2^-100, b] of several divisors and for random (a, b) pairs
// (tests/test_gpu_quotient.py). Here a / b >= 2^-25 or a = 0 (a = x + hx with
// |x| <= hx). Measured: -0.8 % per photon-step on the batch (FAST), -1.6 % (EXACT).
__device__ __forceinline__ float quot_rn(float a, float b, float y) {
  const float q0 = a * y;
  const float q1 = fmaf(fmaf(-q0, b, a), y, q0);
  return fmaf(fmaf(-q1, b, a), y, q1);
}
__device__ __forceinline__ uint32_t xy_bin(float x, float y, const DevParams& P, uint32_t xy_bins) {
  const float nbf = static_cast<float>(xy_bins);
  const uint32_t ix = static_cast<uint32_t>(fminf(quot_rn(x + P.hx, 2.0f * P.hx, P.inv2hx) * nbf, nbf - 1.0f));
  const uint32_t iy = static_cast<uint32_t>(fminf(quot_rn(y + P.hy, 2.0f * P.hy, P.inv2hy) * nbf, nbf - 1.0f));
  return iy * xy_bins + ix;
}

}  // namespace optx
