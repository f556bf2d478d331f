// Checks the branch-free arithmetic of the photon step
// (gpu_optical_photons_b200/csrc/optx_device.cuh) against the IEEE operations it
// stands for: m_sqrt and m_rcp for every float of their ranges, m_div for random
// and extreme mantissa pairs, to_uniform for every word, fresnel_reflects against
// u <= fresnel_R, box_exit against box_exit_ieee. Prints one line per check and
// exits non-zero on a mismatch. `all-pairs` as the first argument checks m_div for
// every pair of mantissas instead. Built and run by tests/test_gpu_ieee.py.
#include <cstdint>
#include <cstdio>
#include <cstring>

#include <cuda_runtime.h>

#include "optx_device.cuh"

namespace {

using namespace optx;

__device__ __forceinline__ uint32_t mix(uint64_t i, uint32_t salt) {  // murmur3 finaliser
  uint64_t h = i * 0x9E3779B97F4A7C15ull + salt * 0xD1B54A32D192ED03ull;
  h ^= h >> 33;
  h *= 0xff51afd7ed558ccdull;
  h ^= h >> 33;
  h *= 0xc4ceb9fe1a85ec53ull;
  h ^= h >> 33;
  return static_cast<uint32_t>(h);
}
__device__ __forceinline__ float unit(uint64_t i, uint32_t salt) { return to_uniform(mix(i, salt)); }
__device__ __forceinline__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }

struct Sqrt {  // i: bits of x
  __device__ bool operator()(uint64_t i) const {
    const float x = __uint_as_float(static_cast<uint32_t>(i));
    return same(m_sqrt(x), __fsqrt_rn(x));
  }
};
struct Rcp {
  __device__ bool operator()(uint64_t i) const {
    const float x = __uint_as_float(static_cast<uint32_t>(i));
    return same(m_rcp(x), __frcp_rn(x)) && same(m_rcp(-x), __frcp_rn(-x));
  }
};
struct Uniform {
  __device__ bool operator()(uint64_t i) const {
    const uint32_t b = static_cast<uint32_t>(i);
    return same(to_uniform(b), __uint2float_rn((b >> 8) + 1u) * (1.0f / 16777216.0f));
  }
};
struct Pair {  // every pair of mantissas: a, b in [1, 2)
  __device__ bool operator()(uint64_t i) const {
    const float a = __uint_as_float(0x3f800000u | static_cast<uint32_t>(i & 0x7fffffu));
    const float b = __uint_as_float(0x3f800000u | static_cast<uint32_t>(i >> 23));
    return same(m_div(a, b), __fdiv_rn(a, b));
  }
};
// Random mantissas and signs, |b| in [2^-60, 2), |a| in [2^-64, 2^20); every fourth
// pair has a mantissa of b next to 1 or 2 (the hardest reciprocals).
struct Div {
  __device__ bool operator()(uint64_t i) const {
    const uint32_t ra = mix(i, 1), rb = mix(i, 2), rc = mix(i, 3);
    uint32_t mb = rb & 0x7fffffu;
    if ((i & 3u) == 0u) mb = (i & 4u) ? 0x7fffffu - (mb & 15u) : (mb & 15u);
    const float a = __uint_as_float((ra & 0x807fffffu) | ((127u - 64u + (rc & 0xffffu) % 84u) << 23));
    const float b = __uint_as_float((rb & 0x80000000u) | mb | ((127u - 60u + (rc >> 16) % 61u) << 23));
    return same(m_div(a, b), __fdiv_rn(a, b)) && m_div(0.0f, b) == 0.0f;
  }
};
struct Fresnel {
  __device__ bool operator()(uint64_t i) const {
    const float n1 = 1.0f + unit(i, 1), n2 = (i & 1u) ? 1.0f : ((i & 2u) ? 1.5f : 0.8f + 1.4f * unit(i, 2));
    volatile float e = n1 / n2;
    const float eta2 = e * e;
    float c = unit(i, 3);
    if ((i & 12u) == 4u && eta2 > 1.0f)  // around the critical angle
      c = sqrtf(fmaxf(0.0f, 1.0f - 1.0f / eta2)) * (1.0f + (unit(i, 4) - 0.5f) * exp2f(-2.0f - 20.0f * unit(i, 5)));
    if ((i & 12u) == 8u) c *= 1e-4f;
    c = fminf(c, 1.0f);
    const float R = fresnel_R(n1, n2, eta2, c);
    float u = unit(i, 6);
    if (i & 16u) u = R * (1.0f + (unit(i, 7) - 0.5f) * exp2f(-24.0f * unit(i, 8)));  // around R
    u = fminf(1.0f, fmaxf(u, 0x1p-24f));
    return fresnel_reflects(n1, n2, eta2, c, u, kOrdinary) == (u <= R);
  }
};
struct Box {
  __device__ bool operator()(uint64_t i) const {
    StepParams P{};
    P.hx = (i & 1u) ? 25.0f : 0.01f + 200.0f * unit(i, 1);
    P.hy = (i & 1u) ? 25.0f : 0.01f + 200.0f * unit(i, 2);
    P.hz = (i & 2u) ? P.hx : 0.01f + 200.0f * unit(i, 3);
    Photon s{};
    const float out = (i & 28u) == 4u ? 1.5f : 1.0f;  // some positions outside the box
    s.px = P.hx * out * (2.0f * unit(i, 4) - 1.0f);
    s.py = P.hy * out * (2.0f * unit(i, 5) - 1.0f);
    s.pz = P.hz * out * (2.0f * unit(i, 6) - 1.0f);
    const float ct = 2.0f * unit(i, 7) - 1.0f, st = sqrtf(fmaxf(0.0f, 1.0f - ct * ct));
    float sp, cp;
    sincosf(6.2831853f * unit(i, 8), &sp, &cp);
    s.dx = st * cp;
    s.dy = st * sp;
    s.dz = ct;
    const uint32_t m = mix(i, 9);
    if ((m & 3u) == 0u) s.px = (m & 4u) ? P.hx : -P.hx;  // on a face
    if ((m & 24u) == 0u) s.dz = (m & 32u) ? 0.0f : -0.0f;
    if ((m & 192u) == 0u) s.dx = (m & 256u) ? 0.0f : -0.0f;
    if ((m & 1536u) == 0u) { s.dy = s.dx; s.py = s.px; }  // ties
    if (s.dx == 0.0f && s.dy == 0.0f && s.dz == 0.0f) s.dy = 1.0f;
    Hit h0{}, h1{};
    const float d0 = box_exit(P, kOrdinary, s, h0), d1 = box_exit_ieee(P, s, h1);
    return same(fmaxf(d0, 0.0f), fmaxf(d1, 0.0f)) && h0.code() == h1.code() && same(h0.along, h1.along) &&
           h0.x == h1.x && h0.y == h1.y && h0.z == h1.z && Hit::of(h0.code(), s).along == h0.along;
  }
};

struct Log {  // i: a word's upper 24 bits
  __device__ bool operator()(uint64_t i) const {
    const float u = to_uniform(static_cast<uint32_t>(i) << 8), l = -m_log(u), g = lg2_approx(u);
    return log_lo(g) <= l && l <= log_hi(g);
  }
};

template <class F>
__global__ void check(F f, uint64_t lo, uint64_t hi, unsigned long long* bad) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  unsigned long long n = 0;
  for (uint64_t i = lo + static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < hi; i += stride)
    n += f(i) ? 0u : 1u;
  if (n) atomicAdd(bad, n);
}

uint64_t bits(float x) {
  uint32_t b;
  std::memcpy(&b, &x, 4);
  return b;
}

template <class F>
int run(const char* name, F f, uint64_t lo, uint64_t hi, unsigned long long* bad) {
  unsigned long long n = 0;
  cudaMemset(bad, 0, sizeof(n));
  check<<<148 * 16, 256>>>(f, lo, hi, bad);
  const cudaError_t err = cudaMemcpy(&n, bad, sizeof(n), cudaMemcpyDeviceToHost);
  std::printf("%s: %llu cases, %llu mismatches (%s)\n", name, static_cast<unsigned long long>(hi - lo), n,
              cudaGetErrorString(err));
  return (n != 0ull || err != cudaSuccess) ? 1 : 0;
}

}  // namespace

int main(int argc, char** argv) {
  unsigned long long* bad = nullptr;
  if (cudaMalloc(&bad, sizeof(unsigned long long)) != cudaSuccess) return 2;
  int rc = 0;
  if (argc > 1 && std::strcmp(argv[1], "all-pairs") == 0) {
    for (uint64_t k = 0; k < 64; ++k)  // in parts of about a second
      rc |= run("m_div, every pair", Pair{}, k << 40, (k + 1) << 40, bad);
  } else {
    rc |= run("m_sqrt", Sqrt{}, bits(0x1p-60f), bits(0x1p60f) + 1, bad);
    rc |= run("m_sqrt(0)", Sqrt{}, 0, 1, bad);
    rc |= run("m_rcp", Rcp{}, bits(0x1p-100f), bits(0x1p100f) + 1, bad);
    rc |= run("log bounds", Log{}, 0, 1ull << 24, bad);
    rc |= run("to_uniform", Uniform{}, 0, 1ull << 32, bad);
    rc |= run("m_div", Div{}, 0, 1ull << 32, bad);
    rc |= run("fresnel_reflects", Fresnel{}, 0, 1ull << 30, bad);
    rc |= run("box_exit", Box{}, 0, 1ull << 30, bad);
  }
  cudaFree(bad);
  return rc;
}
