// Device check of fc3dgpu_ieee64.cuh: division, square root and comparisons
// against the device's own IEEE operations on edge and random operands, and the
// largest errors of the approximate seeds over every mantissa, in units of the
// last place.  Prints the number of mismatches, then the reciprocal's and the
// reciprocal root's largest seed error.
#include <cstdio>

#include "fc3dgpu_ieee64.cuh"
using namespace fc3dgpu;

struct Result {
  unsigned long long bad;
  unsigned rcp, rsqrt;  // in 1/1024 units of the last place, rounded up
};

__device__ uint64_t mix(uint64_t x) {
  x += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return x ^ (x >> 31);
}
__device__ bool differ(double x, double y) { return ie_bits(x) != ie_bits(y) && !(x != x && y != y); }

__device__ int check(double x, double y) {
  int bad = differ(ie_div(x, y), x / y) + differ(ie_sqrt(x), sqrt(x)) + differ(ie_sqrt(ie_abs(x)), sqrt(ie_abs(x)));
  double q0, q1;
  ie_div2(x, y, ie_den(y), q0, q1);
  bad += differ(q0, x / y) + differ(q1, y / y);
  bad += (ie_lt(x, y) != (x < y)) + (ie_le(x, y) != (x <= y)) + (ie_positive(x) != (x > 0)) + (ie_nan(x) != (x != x));
  const double a = ie_abs(x), b = ie_abs(y);
  bad += (ie_lt_pos(a, b) != (a < b)) + (ie_le_pos(a, b) != (a <= b));
  return bad;
}

__device__ const uint64_t edge[] = {
    0x0000000000000000, 0x8000000000000000, 0x3ff0000000000000, 0xbff0000000000000,  // 0, -0, 1, -1
    0x7ff0000000000000, 0xfff0000000000000, 0x7ff8000000000000, 0xfff8000000000000,  // infinities, NaN
    0x0000000000000001, 0x8000000000000001, 0x000fffffffffffff, 0x0010000000000000,  // subnormal to normal
    0x0010000000000001, 0x001fffffffffffff, 0x7fefffffffffffff, 0xffefffffffffffff,  // smallest, largest
    0x3fffffffffffffff, 0x3ff0000000000001, 0x4000000000000000, 0x4008000000000000,  // about 2, 1, 3
    0x3fe0000000000000, 0x3fefffffffffffff, 0x0020000000000000, 0x7fe0000000000000};
constexpr int EDGES = sizeof(edge) / sizeof(edge[0]);

__global__ void k_values(long long n, Result* out) {
  int bad = 0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    uint64_t a, b;
    if (i < EDGES * EDGES) {
      a = edge[i / EDGES];
      b = edge[i % EDGES];
    } else {
      a = mix(2 * i);
      b = mix(2 * i + 1);
      const int k = i & 15;
      const uint64_t mantissa = 0xfffffffffffffull;
      if (k == 1) a &= ~mantissa;
      if (k == 2) b &= ~mantissa;
      if (k == 3) a |= mantissa;
      if (k == 4) b |= mantissa;
      if (k == 5) b = (b & ~mantissa) | (mix(i) & 0xff);
      if (k == 6) a &= 0x800fffffffffffffull;                                    // subnormal
      if (k == 7) b = ((a & mantissa) | (b & ~mantissa)) + mix(i) % 5 - 2;       // quotients next to a power of two
      if (k >= 8) {
        a = (a & 0x800fffffffffffffull) | ((1003 + mix(i) % 40) << 52);
        b = (b & 0x800fffffffffffffull) | ((1003 + mix(~i) % 40) << 52);
      }
    }
    bad += check(ie_double(a), ie_double(b));
    double z = ie_double((b & 0xfffffffffffffull) | ((1000 + mix(i) % 50) << 52));  // next to a square
    z = ie_double(ie_bits(z * z) + mix(i) % 5 - 2);
    bad += differ(ie_sqrt(z), sqrt(z));
  }
  if (bad) atomicAdd(&out->bad, (unsigned long long)bad);
}

// every FP32 in [1, 2) for the reciprocal, in [1, 4) for the reciprocal root;
// both results lie in [1/2, 1], where a unit is 2^-24
__global__ void k_seeds(Result* out) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < 3u << 23; i += gridDim.x * blockDim.x) {
    const unsigned f = 0x3f800000u + (i >> 23 == 0 ? i : i - (1u << 23));
    const double x = (double)__uint_as_float(f);
    const double e = i >> 23 == 0 ? (double)__uint_as_float(ie_rcp_seed(f)) - 1.0 / x
                                  : (double)__uint_as_float(ie_rsqrt_seed(f)) - 1.0 / sqrt(x);
    atomicMax(i >> 23 == 0 ? &out->rcp : &out->rsqrt, (unsigned)ceil(fabs(e) * 0x1p24 * 1024.0));
  }
}

int main() {
  Result* r = nullptr;
  if (cudaMallocManaged(&r, sizeof(Result)) != cudaSuccess) return 2;
  *r = Result{0, 0, 0};
  k_values<<<608, 128>>>(1 << 24, r);
  k_seeds<<<608, 128>>>(r);
  if (cudaDeviceSynchronize() != cudaSuccess) return 3;
  std::printf("%llu %.3f %.3f\n", r->bad, r->rcp / 1024.0, r->rsqrt / 1024.0);
  return 0;
}
