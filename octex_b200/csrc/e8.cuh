// E8 lattice decode and 64-bit cell code, shared by every kernel that needs a cell.
//
// Semantics follow the reference's device functions (hpdic/octex,
// cpp/src/neighbors/octex/detail/e8.cuh:25-85): E8 = D8 u (D8 + 1/2); the nearest D8 point is the
// coordinate-wise rounding (half to even) with the worst-rounded coordinate moved one step when
// the sum is odd; the nearer of the two cosets wins, the integer one on a tie; the code is a
// prime-weighted sum of the doubled coordinates per block, chained over blocks with the 64-bit
// golden-ratio constant and finished by two xor-shift-multiply steps.
//
// Floating-point contract: every operation is written with explicit round-to-nearest intrinsics so
// that the compiler cannot fuse or reorder them; the only fused multiply-adds are the two
// squared-error accumulations, one per coordinate in coordinate order. The CPU checker of this
// repository states the same contract, which makes codes comparable bit for bit.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace octex_b200 {

static __device__ __constant__ unsigned long long kCellPrimes[8] = {1000003ULL,
                                                              998244353ULL,
                                                              1000000007ULL,
                                                              2147483647ULL,
                                                              1099511627791ULL,
                                                              4398042316799ULL,
                                                              70368744177643ULL,
                                                              1125899906842597ULL};
constexpr unsigned long long kGolden = 0x9E3779B97F4A7C15ULL;

/// Nearest D8 point of v[0..8) into out[0..8).
__device__ __forceinline__ void nearest_d8(const float (&v)[8], float (&out)[8])
{
  float total = 0.f, worst = -1.f, worst_e = 0.f;
  int worst_at = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const float r = rintf(v[i]);
    out[i]        = r;
    total         = __fadd_rn(total, r);
    const float e = __fsub_rn(v[i], r);
    const float a = fabsf(e);
    if (a > worst) {
      worst    = a;
      worst_at = i;
      worst_e  = e;
    }
  }
  // total is an integer-valued float: odd <=> its remainder by 2 is non-zero
  if (fmodf(total, 2.f) != 0.f) {
    const float step = worst_e >= 0.f ? 1.f : -1.f;
#pragma unroll
    for (int i = 0; i < 8; i++)
      if (i == worst_at) out[i] = __fadd_rn(out[i], step);
  }
}

/// Nearest E8 point of v[0..8) into out[0..8) (coordinates in Z/2).
__device__ __forceinline__ void nearest_e8(const float (&v)[8], float (&out)[8])
{
  float ints[8], halves[8], moved[8];
#pragma unroll
  for (int i = 0; i < 8; i++)
    moved[i] = __fsub_rn(v[i], 0.5f);
  nearest_d8(v, ints);
  nearest_d8(moved, halves);
  float err_i = 0.f, err_h = 0.f;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    halves[i]     = __fadd_rn(halves[i], 0.5f);
    const float a = __fsub_rn(v[i], ints[i]);
    const float c = __fsub_rn(v[i], halves[i]);
    err_i         = __fmaf_rn(a, a, err_i);
    err_h         = __fmaf_rn(c, c, err_h);
  }
  const bool take_ints = err_i <= err_h;
#pragma unroll
  for (int i = 0; i < 8; i++)
    out[i] = take_ints ? ints[i] : halves[i];
}

/// Prime-weighted sum of the doubled coordinates of the E8 point nearest to v (one block).
__device__ __forceinline__ unsigned long long block_code(const float (&v)[8])
{
  float p[8];
  nearest_e8(v, p);
  unsigned long long hb = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const long long twice = static_cast<long long>(__fmul_rn(2.f, p[i]));
    hb += static_cast<unsigned long long>(twice) * kCellPrimes[i];
  }
  return hb;
}

/// Final mixing of a chained block code.
__device__ __forceinline__ long long finish_code(unsigned long long h)
{
  long long s = static_cast<long long>(h);
  s           = static_cast<long long>(static_cast<unsigned long long>(s ^ (s >> 31)) * kGolden);
  return s ^ (s >> 29);
}

/// Cell code of the 8*B coordinates y scaled by inv_f.
template <int B>
__device__ __forceinline__ long long cell_code(const float (&y)[8 * B], float inv_f)
{
  unsigned long long h = 0;
#pragma unroll
  for (int j = 0; j < B; j++) {
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; i++)
      v[i] = __fmul_rn(y[8 * j + i], inv_f);
    const unsigned long long hb = block_code(v);
    h                           = (j == 0) ? hb : h * kGolden + hb;
  }
  return finish_code(h);
}

// ---------------------------------------------------------------------------------------------
// The same decode for coordinates known to be small: every |v[i]| < kTameLimit (and no NaN). Under
// that bound each step below gives the value the general code gives, so the codes are identical;
// what changes is the instruction mix: no conversion-unit instructions and no branches.
//   * rint(x) = (x + 1.5 * 2^23) - 1.5 * 2^23 in round-to-nearest arithmetic (ties to even), exact
//     for |x| < 2^22. A rounded -0 comes out as +0, which no later step can tell apart.
//   * the sum of the rounded coordinates is an exact integer below 2^24: it is odd iff half of it is
//     not an integer.
//   * 2 p + 1.5 * 2^23 is exact, and its bit pattern is 0x4B400000 + 2 p as an integer: the weighted
//     sum runs over these unsigned words and the constant part is taken off at the end (all modulo
//     2^64, as in the general code).
constexpr float kTameLimit = 1048576.f;  // 2^20
constexpr float kRintMagic = 12582912.f;  // 1.5 * 2^23, bit pattern 0x4B400000

__host__ __device__ constexpr unsigned long long cell_prime(int i)
{
  return i == 0   ? 1000003ULL
         : i == 1 ? 998244353ULL
         : i == 2 ? 1000000007ULL
         : i == 3 ? 2147483647ULL
         : i == 4 ? 1099511627791ULL
         : i == 5 ? 4398042316799ULL
         : i == 6 ? 70368744177643ULL
                  : 1125899906842597ULL;
}

__device__ __forceinline__ float rint_tame(float x)
{
  return __fsub_rn(__fadd_rn(x, kRintMagic), kRintMagic);
}

__device__ __forceinline__ void nearest_d8_tame(const float (&v)[8], float (&out)[8])
{
  out[0]        = rint_tame(v[0]);
  float total   = out[0];
  float worst_e = __fsub_rn(v[0], out[0]);
  int worst_at  = 0;
#pragma unroll
  for (int i = 1; i < 8; i++) {
    const float r = rint_tame(v[i]);
    out[i]        = r;
    total         = __fadd_rn(total, r);
    const float e = __fsub_rn(v[i], r);
    if (fabsf(e) > fabsf(worst_e)) {  // strictly larger: the first of equal errors stays
      worst_at = i;
      worst_e  = e;
    }
  }
  const float half = __fmul_rn(total, 0.5f);
  const bool odd   = rint_tame(half) != half;
  const float step = odd ? (worst_e >= 0.f ? 1.f : -1.f) : 0.f;
#pragma unroll
  for (int i = 0; i < 8; i++)
    out[i] = __fadd_rn(out[i], i == worst_at ? step : 0.f);
}

__device__ __forceinline__ unsigned long long block_code_tame(const float (&v)[8])
{
  float ints[8], halves[8], moved[8];
#pragma unroll
  for (int i = 0; i < 8; i++)
    moved[i] = __fsub_rn(v[i], 0.5f);
  nearest_d8_tame(v, ints);
  nearest_d8_tame(moved, halves);
  float err_i = 0.f, err_h = 0.f;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    halves[i]     = __fadd_rn(halves[i], 0.5f);
    const float a = __fsub_rn(v[i], ints[i]);
    const float c = __fsub_rn(v[i], halves[i]);
    err_i         = __fmaf_rn(a, a, err_i);
    err_h         = __fmaf_rn(c, c, err_h);
  }
  const bool take_ints = err_i <= err_h;
  unsigned long long hb = 0, primes = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const float p    = take_ints ? ints[i] : halves[i];
    const unsigned u = __float_as_uint(__fmaf_rn(2.f, p, kRintMagic));
    hb += static_cast<unsigned long long>(u) * cell_prime(i);
    primes += cell_prime(i);
  }
  return hb - 0x4B400000ULL * primes;
}

/// cell_code for coordinates with |y[i] * inv_f| < kTameLimit: the same code, fewer instructions.
template <int B>
__device__ __forceinline__ long long cell_code_tame(const float (&y)[8 * B], float inv_f)
{
  unsigned long long h = 0;
#pragma unroll
  for (int j = 0; j < B; j++) {
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; i++)
      v[i] = __fmul_rn(y[8 * j + i], inv_f);
    const unsigned long long hb = block_code_tame(v);
    h                           = (j == 0) ? hb : h * kGolden + hb;
  }
  return finish_code(h);
}

// ---------------------------------------------------------------------------------------------
// The same code again with about half the arithmetic of block_code_tame (one coset repaired instead of two),
// for the kernel that decodes every query. Rounding v to r leaves e = v - r (exact); the other coset leaves
// 1/2 - |e| in every coordinate. With A = sum |e|, m = max |e|, n = min |e| the squared errors of the
// two cosets after their parity repairs differ by
//     D = A - 2 + (odd ? 1 - 2 m : 0) - (odd' ? 2 n : 0)
// so the nearer coset is known before either is worked out, and only the one taken is repaired. D is
// good to 4e-6 (eight additions of terms up to 1/2), and the two sums that block_code_tame compares, of
// at most eight squares up to 1, to 1e-6 each. What grows with the coordinates is the rounding of
// v - 1/2, which the half coset starts from: exact for v >= 1/2, but a v just above -2^k crosses a
// binade, so it is off by up to d = (V + 1/2) 2^-24 where no |v| exceeds V. A coordinate within d of a
// tie may then be rounded the other way (its squared error changes by 2 d, in all eight at worst), and
// the coordinate repaired may be one within 2 d of the worst (4 d), or one of those at a tie (2 d): 22 d
// in all. Where |D| is below decode_margin = 2.1e-5 + V 2^-19 >= 6e-6 + 22 d the block is `doubtful`
// and goes to block_code_tame. The rest is exact: both parities come
// from the low bits of the rounded values, and the coset taken is rounded and repaired by the same
// operations on the same values as in nearest_d8_tame. Two coordinates at a time share an instruction
// (the packed fp32 arithmetic of sm_100, each half rounded as on its own).

struct f32_pair {
  unsigned long long v;
};
__device__ __forceinline__ f32_pair pack2(float lo, float hi)
{
  f32_pair p;
  asm("mov.b64 %0, {%1, %2};" : "=l"(p.v) : "f"(lo), "f"(hi));
  return p;
}
__device__ __forceinline__ void unpack2(f32_pair p, float& lo, float& hi)
{
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(p.v));
}
__device__ __forceinline__ f32_pair add2(f32_pair a, f32_pair b)
{
  f32_pair d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
  return d;
}
__device__ __forceinline__ f32_pair mul2(f32_pair a, f32_pair b)
{
  f32_pair d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
  return d;
}
__device__ __forceinline__ f32_pair fma2(f32_pair a, f32_pair b, f32_pair c)
{
  f32_pair d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return d;
}
__device__ __forceinline__ float max3_abs(float a, float b, float c)
{
  return fmaxf(fmaxf(fabsf(a), fabsf(b)), fabsf(c));
}
__device__ __forceinline__ float min3_abs(float a, float b, float c)
{
  return fminf(fminf(fabsf(a), fabsf(b)), fabsf(c));
}

/// The larger magnitude, NaN when either is none (fmaxf would drop it).
__device__ __forceinline__ float max_abs_nan(float a, float b)
{
  float d;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(fabsf(a)), "f"(fabsf(b)));
  return d;
}

/// Below this |D| a block with no coordinate beyond `reach` (before the scaling by inv) is doubtful.
__device__ __forceinline__ float decode_margin(float reach, float inv) { return fmaf(reach * inv, 1.9073486e-6f, 2.1e-5f); }

/// Block code of the four pairs y scaled by inv; primes: the eight cell primes in shared memory;
/// margin: decode_margin of the block.
__device__ __forceinline__ unsigned long long block_code_fast(const f32_pair (&y)[4], float inv, float margin,
                                                              const unsigned long long* primes, bool& doubtful)
{
  const f32_pair up = pack2(kRintMagic, kRintMagic), down = pack2(-kRintMagic, -kRintMagic);
  const f32_pair minus1 = pack2(-1.f, -1.f), less_half = pack2(-0.5f, -0.5f), scale = pack2(inv, inv);
  f32_pair v[4];
  float e[8], M[8], H[8];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    v[i]             = mul2(y[i], scale);
    const f32_pair b = add2(v[i], up);
    const f32_pair d = fma2(add2(b, down), minus1, v[i]);
    const f32_pair h = add2(add2(v[i], less_half), up);
    unpack2(b, M[2 * i], M[2 * i + 1]);
    unpack2(d, e[2 * i], e[2 * i + 1]);
    unpack2(h, H[2 * i], H[2 * i + 1]);
  }
  unsigned odd_i = 0, odd_h = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    odd_i ^= __float_as_uint(M[i]);
    odd_h ^= __float_as_uint(H[i]);
  }
  const float A = ((fabsf(e[0]) + fabsf(e[1])) + (fabsf(e[2]) + fabsf(e[3]))) +
                  ((fabsf(e[4]) + fabsf(e[5])) + (fabsf(e[6]) + fabsf(e[7])));
  const float m = fmaxf(max3_abs(e[0], e[1], e[2]), fmaxf(max3_abs(e[3], e[4], e[5]), fmaxf(fabsf(e[6]), fabsf(e[7]))));
  const float n = fminf(min3_abs(e[0], e[1], e[2]), fminf(min3_abs(e[3], e[4], e[5]), fminf(fabsf(e[6]), fabsf(e[7]))));
  float D = A - 2.f;
  if (odd_i & 1u) D += fmaf(-2.f, m, 1.f);
  if (odd_h & 1u) D = fmaf(-2.f, n, D);
  doubtful         = fabsf(D) < margin;
  const bool halves = D > 0.f;
  const bool odd    = ((halves ? odd_h : odd_i) & 1u) != 0;
  // the coset taken, from its own rounding on
  const f32_pair off = halves ? less_half : pack2(0.f, 0.f);
  float c[8];
  unsigned long long sum = 0;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const f32_pair w = add2(v[i], off);
    const f32_pair b = add2(w, up);
    const f32_pair d = fma2(add2(b, down), minus1, w);
    unpack2(d, c[2 * i], c[2 * i + 1]);
    float lo, hi;
    unpack2(b, lo, hi);
    sum += static_cast<unsigned long long>(__float_as_uint(lo)) * cell_prime(2 * i);
    sum += static_cast<unsigned long long>(__float_as_uint(hi)) * cell_prime(2 * i + 1);
  }
  // the worst rounded coordinate, the first of equal ones: a tree in which the left side stays unless
  // the right one is strictly larger
  int at[8];
#pragma unroll
  for (int i = 0; i < 8; i++)
    at[i] = i;
#pragma unroll
  for (int s = 1; s < 8; s <<= 1)
#pragma unroll
    for (int i = 0; i < 8; i += 2 * s) {
      const bool right = fabsf(c[i + s]) > fabsf(c[i]);
      c[i]             = right ? c[i + s] : c[i];
      at[i]            = right ? at[i + s] : at[i];
    }
  const unsigned long long prime = primes[at[0]];
  unsigned long long step        = c[0] >= 0.f ? prime : 0ULL - prime;
  step                           = odd ? step : 0ULL;
  constexpr unsigned long long all = cell_prime(0) + cell_prime(1) + cell_prime(2) + cell_prime(3) + cell_prime(4) +
                                     cell_prime(5) + cell_prime(6) + cell_prime(7);
  // twice the coordinates: 2 (bits - 0x4B400000), plus 1 in the half coset
  const unsigned long long constant = halves ? all - 2 * 0x4B400000ULL * all : 0ULL - 2 * 0x4B400000ULL * all;
  return 2 * (sum + step) + constant;
}

}  // namespace octex_b200
