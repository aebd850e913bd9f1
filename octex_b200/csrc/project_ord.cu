// Projection of a query batch in dimension order with the E8 decode and the cell lookup in the same
// kernel (sm_100a), for indexes whose copies do not have the four blocks the tensor-core kernel
// works on: centring, Y = half(fp32(half(q - mean) . ut^T) + shift), cell codes and lookup, and the
// sketch-space queries in extra blocks (hpdic/octex, cpp/src/neighbors/octex/search.cu:303-341,
// detail/search_kernels.cuh:57-69,100-126). Every dot product takes one fused multiply-add per
// dimension in dimension order, as in project_ordered_kernel and the CPU checker, so the coordinates
// are theirs bit for bit.
//
// A block of 256 threads makes 64 rows x up to 64 columns (whole copies), 4 x 4 sums per thread, from
// operands staged in shared memory in steps of 32 dimensions, the next step's loads in flight behind
// the sums; the coordinates stay in shared memory, where each (query, copy) is decoded. One launch
// replaces four (centring, projection, codes, lookup): 300 queries x 8 copies x 48 dimensions took
// 57 us in them.

#include "kernels.hpp"

#include "prep_common.cuh"

#include <algorithm>

namespace octex_b200::kernels {

namespace {

constexpr int kRows = 64, kStep = 32, kLd = kRows + 4;

template <int B>
struct ord_shape {
  static constexpr int kC = 8 * B <= 64 ? 64 / (8 * B) : 1;  // copies per block
  static constexpr int kW = kC * 8 * B;                      // columns per block
};

template <int B>
__global__ void __launch_bounds__(256) project_lookup_kernel(const sketch_job job, int sk_blocks, int per_block,
                                                             const __half* __restrict__ ut, int ldu, int Cg, int L,
                                                             const __half* __restrict__ shift,
                                                             const float* __restrict__ inv_f, float tame_y,
                                                             const tc_lookup look)
{
  constexpr int kC = ord_shape<B>::kC, kW = ord_shape<B>::kW, kYd = 8 * B + 4;
  constexpr int kPairs    = kRows * kC;
  constexpr int kStaging  = 2 * kStep * kLd;
  constexpr int kLookup   = kPairs * (kYd + 1) + 512;
  constexpr int kMost     = kStaging > kLookup ? kStaging : kLookup;
  __shared__ __align__(16) float smem[kMost > sketch_tile<1>::kWords ? kMost : sketch_tile<1>::kWords];
  let_next_kernel_start();
  if (static_cast<int>(blockIdx.x) < sk_blocks) {
    sketch_block<1>(job, blockIdx.x, smem);
    return;
  }
  __shared__ cell_level lv[kC * 16];
  __shared__ unsigned long long primes[8];
  float* sa = smem;               // [32 dims][68 rows]
  float* sb = smem + kStep * kLd;  // [32 dims][68 columns]
  const int tiles = (Cg + kC - 1) / kC;
  const int c0    = ((blockIdx.x - sk_blocks) % tiles) * kC;
  const int row0  = ((blockIdx.x - sk_blocks) / tiles) * per_block;
  const int m = job.m, D = job.D, N = Cg * 8 * B, col0 = c0 * 8 * B;
  const int rows = min(per_block, m - row0);
  fill_primes(primes);
  if (threadIdx.x < kC * L) lv[threadIdx.x] = c0 + threadIdx.x / L < Cg ? look.levels[c0 * L + threadIdx.x] : cell_level{0, 0, -1, 0};
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  float x[8];
  uint4 w;
  auto fetch = [&](int d0) {
#pragma unroll
    for (int u = 0; u < 8; u++) {
      const int i = threadIdx.x + u * 256, r = i / kStep, d = d0 + i % kStep;
      x[u] = r < rows && d < D ? __ldg(job.q + static_cast<int64_t>(row0 + r) * D + d) : 0.f;
    }
    const int col = threadIdx.x >> 2, k = (threadIdx.x & 3) * 8;
    w = make_uint4(0, 0, 0, 0);  // rows of ut are padded with zeros up to a multiple of 64
    if (col < kW && col0 + col < N)
      w = __ldg(reinterpret_cast<const uint4*>(ut + static_cast<int64_t>(col0 + col) * ldu + d0 + k));
  };
  float acc[4][4] = {};
  fetch(0);
  for (int d0 = 0; d0 < D; d0 += kStep) {
    const int mine = threadIdx.x % kStep;
    const float mu = d0 + mine < D ? __ldg(job.mean + d0 + mine) : 0.f;
#pragma unroll
    for (int u = 0; u < 8; u++) {
      const int r = (threadIdx.x + u * 256) / kStep;
      if (r < rows) sa[mine * kLd + r] = __half2float(__float2half_rn(__fsub_rn(x[u], mu)));
    }
    {
      const int col = threadIdx.x >> 2, k = (threadIdx.x & 3) * 8;
      const unsigned h2[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int i = 0; i < 4; i++) {
        sb[(k + 2 * i) * kLd + col]     = __half2float(__ushort_as_half(static_cast<unsigned short>(h2[i] & 0xffffu)));
        sb[(k + 2 * i + 1) * kLd + col] = __half2float(__ushort_as_half(static_cast<unsigned short>(h2[i] >> 16)));
      }
    }
    __syncthreads();
    if (d0 + kStep < D) fetch(d0 + kStep);
    if (4 * ty < rows && 4 * tx < kW) {
      const int dd = min(kStep, D - d0);
#pragma unroll 8
      for (int d = 0; d < dd; d++) {
        const float4 a4  = *reinterpret_cast<const float4*>(sa + d * kLd + 4 * ty);
        const float4 b4  = *reinterpret_cast<const float4*>(sb + d * kLd + 4 * tx);
        const float a[4] = {a4.x, a4.y, a4.z, a4.w}, b[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
          for (int j = 0; j < 4; j++)
            acc[i][j] = __fmaf_rn(a[i], b[j], acc[i][j]);
      }
    }
    __syncthreads();
  }
  // coordinates of pair (row, copy) of the block: ys[(row * kC + copy) * kYd ..]
  float* ys = smem;
  int* best = reinterpret_cast<int*>(smem + kPairs * kYd);
  int* hit  = best + kPairs;
  if (4 * tx < kW) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int col  = 4 * tx + j;
      const float sh = col0 + col < N ? __half2float(shift[col0 + col]) : 0.f;
#pragma unroll
      for (int i = 0; i < 4; i++)
        if (4 * ty + i < rows)
          ys[((4 * ty + i) * kC + col / (8 * B)) * kYd + col % (8 * B)] =
            __half2float(__float2half_rn(__fadd_rn(acc[i][j], sh)));
    }
  }
  __syncthreads();
  const int pairs = rows * kC;
  auto coordinates = [&](int p, int sub, f32_pair(&y)[4 * group_decoder<B>::kOwn]) {
    const float* src = ys + p * kYd + sub * 8 * group_decoder<B>::kOwn;
#pragma unroll
    for (int i = 0; i < 2 * group_decoder<B>::kOwn; i++) {
      const float4 v = *reinterpret_cast<const float4*>(src + 4 * i);
      y[2 * i]       = pack2(v.x, v.y);
      y[2 * i + 1]   = pack2(v.z, v.w);
    }
  };
  if (look.stats == nullptr && spread_pays<B>(pairs, L))
    lookup_spread<B, kC>(look, coordinates, best, hit, pairs, tame_y, inv_f, lv, primes, L, row0, c0, Cg);
  else
    lookup_pairs<B, kC>(look, coordinates, pairs, tame_y, inv_f, lv, primes, L, row0, c0, Cg);
}

}  // namespace

auto project_lookup_ordered(const sketch_job& job, int blocks, const __half* ut, int ldu, int copies, int L,
                            const __half* shift, const float* inv_f, float finest, const tc_lookup& look, int sms,
                            cudaStream_t s) -> project_shape
{
  project_shape took{project_form::ordered, 0};
  if (job.m <= 0 || copies <= 0) return took;
  const float tame_y = finest > 0.f ? kTameLimit * finest * 0.99f : 0.f;
  const int sk       = sketch_blocks<1>(job);
  // A block goes through its pairs in turns of 256 lanes, so one of 64 rows takes several times the latency of a turn
  // where there are multiprocessors left for more blocks of fewer: as few rows as give each of them a block, but not
  // fewer than a turn takes with all levels at once. us a search, 64 rows and these: 8 copies x 48 dimensions in two
  // blocks, 64 queries 78 and 71, 300 79.5 and 73.7, 1 000 92 and 87; 64 copies, one round, 100 49 and 43; 20 x 96 in
  // three blocks, 300 51 and 47. The sums of a block take as long for fewer rows: with three blocks for a
  // multiprocessor 64 copies and 1 000 queries take 73 us instead of 62, 40 x 768 dimensions and 300 111 instead of 97.
  auto launch        = [&](auto kernel, int copies_a_block, int group) {
    const int tiles = (copies + copies_a_block - 1) / copies_a_block;
    const int fit   = std::max(1, (sms / job.beside - sk) / tiles);
    const int least = 256 / (group * copies_a_block * std::max(L, 1));
    const int rows  = std::min(kRows, (std::max({(job.m + fit - 1) / fit, least, 1}) + 3) & ~3);
    const unsigned grid = static_cast<unsigned>(sk + tiles * ((job.m + rows - 1) / rows));
    took.rows = rows;
    kernel<<<grid, 256, 0, s>>>(job, sk, rows, ut, ldu, copies, L, shift, inv_f, tame_y, look);
  };
  switch (blocks) {
    case 1: launch(project_lookup_kernel<1>, ord_shape<1>::kC, kGroup<1>); break;
    case 2: launch(project_lookup_kernel<2>, ord_shape<2>::kC, kGroup<2>); break;
    case 3: launch(project_lookup_kernel<3>, ord_shape<3>::kC, kGroup<3>); break;
    case 4: launch(project_lookup_kernel<4>, ord_shape<4>::kC, kGroup<4>); break;
    case 5: launch(project_lookup_kernel<5>, ord_shape<5>::kC, kGroup<5>); break;
    case 6: launch(project_lookup_kernel<6>, ord_shape<6>::kC, kGroup<6>); break;
    case 8: launch(project_lookup_kernel<8>, ord_shape<8>::kC, kGroup<8>); break;
    default: break;  // the loader rejects other block counts
  }
  return took;
}

}  // namespace octex_b200::kernels
