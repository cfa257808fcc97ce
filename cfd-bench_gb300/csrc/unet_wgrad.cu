// Weight gradients of the U-Net's 3x3x3 convolutions: for each tap a GEMM over
// the cells, dW[tap][o][i] = sum G[cell][o] X[cell + tap][i] (M = output
// channels, N = input channels, K = cells), BF16 operands and FP32 sums.
//
// A block takes x-runs of up to 64 cells and marches over rows y. For a row it
// needs the G row once and the nine X rows around it; X rows live in a ring
// of four rows (three planes each) in shared memory, so each step brings in
// three new X rows and one G row by 16-byte cp.async while the step before
// computes, and all 27 taps read what is there. Nine warps, one per (dz, dy),
// each hold the accumulators of its three dx taps for the whole march: the dx
// shift is a row offset of the fragment loads. Both operands are stored with
// the channels contiguous, i.e. K by M and K by N, so ldmatrix.trans gives the
// fragments; the rows are padded by 16 bytes, which spreads eight consecutive
// rows over all banks. The bias gradient is the product with a fragment of
// ones. Blocks write their sums to scratch and k_wgrad_fold adds them in a
// fixed order.
//
// mma.sync, not tcgen05: M is 16 to 32 channels a tile, where tcgen05 takes at
// least 64 rows, so three or four planes of taps would have to share a product;
// the layer is bound by moving fragments, not by the tensor pipe.
//
// Measured on a batch of eight 64^3 volumes: all weight and bias gradients of a
// training step 22.6 -> 1.8 ms (one block per (cells, tap), which read both
// operands 27 times and assembled fragments from 16-bit loads, before).
#include <cuda_bf16.h>

#include <cstdint>

#include "nusif_internal.h"
#include "unet_wgrad.h"

namespace nusif {
namespace {

using bf16 = __nv_bfloat16;

constexpr int kWarps = 9, kThreads = 32 * kWarps;
constexpr int kRun = 64;    // cells of an x-run
constexpr int kSlots = 4;   // X rows y - 1 .. y + 2
constexpr int kWave = 304;  // two blocks on each of 152 SMs

struct Args {
  WgradSrc s0, s1;
  const bf16 *g;
  const float *g32;  // FP32 G of one channel, split into three BF16 channels
  int B, Z, Y, X;
  int run, xt;       // cells of a run, runs per row
  int yc, yt;        // rows of a march, marches per plane
  int items;         // B * Z * xt * yt
  int co;            // G's channels
  int parts_n;       // tiles over the input channels
  int chain;         // cells whose products are summed without rounding, a run at least
  float *partial;    // [part][block][27 * TM * TN + TM]
};

__device__ __forceinline__ uint32_t saddr(const void *p)
{
  return (uint32_t)__cvta_generic_to_shared(p);
}

// 16 bytes to shared memory; zeros where !ok (then nothing is read)
__device__ __forceinline__ void copy16(uint32_t dst, const void *src, bool ok)
{
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src),
      "r"(ok ? 16 : 0) : "memory");
}

__device__ __forceinline__ void ldmatrix_t(uint32_t (&r)[4], uint32_t addr)
{
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}

__device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
      "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <int TM, int TN>
struct Layout {
  static constexpr int kXp = TN * 2 + 16, kGp = TM * 2 + 16;  // bytes per cell
  static constexpr int kXrow = (kRun + 2) * kXp, kGrow = kRun * kGp;
  static constexpr int kSmem = kSlots * 3 * kXrow + 2 * kGrow;
  static constexpr int kXChunks = TN / 8, kGChunks = TM / 8;
  static constexpr int kXPer = (3 * (kRun + 2) * kXChunks + kThreads - 1) / kThreads;
  static constexpr int kGPer = (kRun * kGChunks + kThreads - 1) / kThreads;
};

// G32: G is one FP32 channel, stored as the three BF16 channels whose sum it
// is (24 bits), the other rows of the tile zero.
// ROWS: the tensor core's own FP32 accumulation truncates, so a long chain of
// products drifts (1e-5 of a gradient over two million cells). The first and
// the last layer, whose gradients were plain FP32 sums before, keep a chain to
// one row and add the rows with rounding (2e-7); at 16 x 16 channels that costs
// 155 -> 220 us on two million cells. The bias gradients, one fragment of one
// warp, do so in every layer. In the others a chain has at most a 256th of the
// cells or 512, whose drift is that of the FP32 additions of the blocks' sums
// (7e-7); where a block has more, it adds its sums to those it has stored.
template <int TM, int TN, bool G32, bool ROWS>
__global__ void __launch_bounds__(kThreads) k_wgrad(Args A)
{
  using L = Layout<TM, TN>;
  constexpr int MT = TM / 16, NT = TN / 8;
  extern __shared__ __align__(16) unsigned char smem[];
  unsigned char *const gs = smem + kSlots * 3 * L::kXrow;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int part = blockIdx.y;
  const int m0 = (part / A.parts_n) * TM, n0 = (part % A.parts_n) * TN;
  const int cells = A.run + 2;  // of an X row

  // this thread's chunks of an X row triple and of a G row
  int x_dst[L::kXPer], x_dz[L::kXPer], x_cell[L::kXPer], x_ch[L::kXPer];
#pragma unroll
  for (int q = 0; q < L::kXPer; q++) {
    const int i = tid + q * kThreads;
    const int c = i % L::kXChunks, r = i / L::kXChunks;
    x_cell[q] = r % cells;
    x_dz[q] = r / cells;  // 0 .. 2; 3 and more: none
    x_ch[q] = n0 + 8 * c;
    x_dst[q] = x_dz[q] * L::kXrow + x_cell[q] * L::kXp + 16 * c;
  }

  // fragment addresses of this lane (ldmatrix: matrix lane / 8, row lane % 8)
  const int mat = lane >> 3, mr = lane & 7;
  const uint32_t a_off = (uint32_t)((mr + (mat >> 1) * 8) * L::kGp + (mat & 1) * 16);
  const uint32_t b_off = (uint32_t)((mr + (mat & 1) * 8) * L::kXp + (mat >> 1) * 16);
  const int dz = warp / 3, dy = warp % 3 - 1;

  float acc[3][MT][NT][4], bias[MT][4], bias_sum[MT][2];
  float sum[ROWS ? 3 : 1][ROWS ? MT : 1][ROWS ? NT : 1][4];
  const auto clear = [&] {
#pragma unroll
    for (int t = 0; t < 3; t++)
#pragma unroll
      for (int m = 0; m < MT; m++)
#pragma unroll
        for (int n = 0; n < NT; n++)
#pragma unroll
          for (int e = 0; e < 4; e++) acc[t][m][n][e] = 0.0f;
  };
  // ROWS: the row's products join the sums
  const auto gather = [&] {
    if constexpr (ROWS) {
#pragma unroll
      for (int t = 0; t < 3; t++)
#pragma unroll
        for (int m = 0; m < MT; m++)
#pragma unroll
          for (int n = 0; n < NT; n++)
#pragma unroll
            for (int e = 0; e < 4; e++) sum[t][m][n][e] += acc[t][m][n][e];
      clear();
    }
  };
  // the block's sums so far join those it has stored
  float *const out =
      A.partial + ((int64_t)part * gridDim.x + blockIdx.x) * (27 * TM * TN + TM);
  const int g = lane >> 2, t2 = 2 * (lane & 3);
  int chained = 0;
  bool stored = false;
  const auto store = [&] {
#pragma unroll
    for (int t = 0; t < 3; t++) {
      float *const o = out + (dz * 9 + (dy + 1) * 3 + t) * TM * TN;
#pragma unroll
      for (int m = 0; m < MT; m++)
#pragma unroll
        for (int n = 0; n < NT; n++)
#pragma unroll
          for (int h = 0; h < 2; h++) {
            float2 *const at =
                reinterpret_cast<float2 *>(o + (16 * m + g + 8 * h) * TN + 8 * n + t2);
            float2 v = make_float2(acc[t][m][n][2 * h], acc[t][m][n][2 * h + 1]);
            if (stored) {
              const float2 was = *at;
              v.x += was.x;
              v.y += was.y;
            }
            *at = v;
          }
    }
    stored = true;
    chained = 0;
  };
  const auto gather_bias = [&] {
#pragma unroll
    for (int m = 0; m < MT; m++) {
      bias_sum[m][0] += bias[m][0];
      bias_sum[m][1] += bias[m][2];
#pragma unroll
      for (int e = 0; e < 4; e++) bias[m][e] = 0.0f;
    }
  };
  clear();
  if constexpr (ROWS) {
#pragma unroll
    for (int t = 0; t < 3; t++)
#pragma unroll
      for (int m = 0; m < MT; m++)
#pragma unroll
        for (int n = 0; n < NT; n++)
#pragma unroll
          for (int e = 0; e < 4; e++) sum[t][m][n][e] = 0.0f;
  }
#pragma unroll
  for (int m = 0; m < MT; m++) {
    bias_sum[m][0] = bias_sum[m][1] = 0.0f;
#pragma unroll
    for (int e = 0; e < 4; e++) bias[m][e] = 0.0f;
  }
  if (G32) {  // the rows that stay zero
    for (int i = tid; i < 2 * L::kGrow / 16; i += kThreads)
      reinterpret_cast<uint4 *>(gs)[i] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
  }

  for (int item = blockIdx.x; item < A.items; item += gridDim.x) {
    const int yi = item % A.yt, r1 = item / A.yt;
    const int xi = r1 % A.xt, bz = r1 / A.xt;
    const int z = bz % A.Z, b = bz / A.Z;
    const int x0 = xi * A.run, y0 = yi * A.yc, y1 = min(y0 + A.yc, A.Y);
    const auto load_x = [&](int y) {  // row y of planes z - 1 .. z + 1
      unsigned char *const slot = smem + ((y + 4) & 3) * 3 * L::kXrow;
#pragma unroll
      for (int q = 0; q < L::kXPer; q++) {
        if (x_dz[q] > 2) continue;
        const int zz = z + x_dz[q] - 1, xx = x0 + x_cell[q] - 1;
        const bool ok = zz >= 0 && zz < A.Z && y >= 0 && y < A.Y && xx >= 0 && xx < A.X;
        const bool second = x_ch[q] >= A.s0.c;
        const WgradSrc &s = second ? A.s1 : A.s0;
        const int ch = second ? x_ch[q] - A.s0.c : x_ch[q];
        const int h = s.up;
        const int64_t cell =
            (((int64_t)b * (A.Z >> h) + (zz >> h)) * (A.Y >> h) + (y >> h)) * (A.X >> h) + (xx >> h);
        const bf16 *src = static_cast<const bf16 *>(s.p) + (ok ? cell * s.c + ch : 0);
        copy16(saddr(slot + x_dst[q]), src, ok);
      }
    };
    float gnext = 0.0f;  // G32: this thread's value of the next row
    const auto load_g = [&](int y) {
      const int64_t row = (((int64_t)b * A.Z + z) * A.Y + y) * A.X + x0;
      if (G32) {
        gnext = tid < A.run && x0 + tid < A.X ? A.g32[row + tid] : 0.0f;
        return;
      }
      unsigned char *const slot = gs + (y & 1) * L::kGrow;
#pragma unroll
      for (int q = 0; q < L::kGPer; q++) {
        const int i = tid + q * kThreads;
        const int c = i % L::kGChunks, cell = i / L::kGChunks;
        if (cell >= A.run) continue;
        const bool ok = x0 + cell < A.X;
        copy16(saddr(slot + cell * L::kGp + 16 * c), A.g + (ok ? (row + cell) * A.co + m0 + 8 * c : 0),
            ok);
      }
    };
    const auto store_g32 = [&](int y) {
      if (tid >= A.run) return;
      bf16 *const d = reinterpret_cast<bf16 *>(gs + (y & 1) * L::kGrow + tid * L::kGp);
      const bf16 hi = __float2bfloat16_rn(gnext);
      const float r = gnext - __bfloat162float(hi);
      const bf16 mid = __float2bfloat16_rn(r);
      d[0] = hi;
      d[1] = mid;
      d[2] = __float2bfloat16_rn(r - __bfloat162float(mid));
    };
    __syncthreads();  // the march before this one is done with the slots
    load_x(y0 - 1);
    load_x(y0);
    load_x(y0 + 1);
    load_g(y0);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    for (int y = y0; y < y1; y++) {
      if (G32) store_g32(y);
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
      __syncthreads();
      if (y + 1 < y1) {
        load_x(y + 2);
        load_g(y + 1);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
      }
      const uint32_t g_row = saddr(gs + (y & 1) * L::kGrow) + a_off;
      const uint32_t x_row = saddr(smem + (((y + dy + 4) & 3) * 3 + dz) * L::kXrow) + b_off;
      for (int k = 0; k < A.run; k += 16) {
        uint32_t a[MT][4];
#pragma unroll
        for (int m = 0; m < MT; m++) ldmatrix_t(a[m], g_row + k * L::kGp + m * 32);
        if (warp == 4) {
#pragma unroll
          for (int m = 0; m < MT; m++) mma(bias[m], a[m], 0x3f803f80u, 0x3f803f80u);
        }
#pragma unroll
        for (int t = 0; t < 3; t++)
#pragma unroll
          for (int n = 0; n < NT; n += 2) {
            uint32_t w[4];
            ldmatrix_t(w, x_row + (k + t) * L::kXp + n * 16);
#pragma unroll
            for (int m = 0; m < MT; m++) {
              mma(acc[t][m][n], a[m], w[0], w[1]);
              mma(acc[t][m][n + 1], a[m], w[2], w[3]);
            }
          }
      }
      if (warp == 4) gather_bias();
      gather();
      chained += A.run;
      if (!ROWS && chained + A.run > A.chain) {
        store();
        clear();
      }
    }
  }
  if constexpr (ROWS) {
#pragma unroll
    for (int t = 0; t < 3; t++)
#pragma unroll
      for (int m = 0; m < MT; m++)
#pragma unroll
        for (int n = 0; n < NT; n++)
#pragma unroll
          for (int e = 0; e < 4; e++) acc[t][m][n][e] = sum[t][m][n][e];
  }
  if (!stored || chained > 0) store();
  if (warp == 4 && (lane & 3) == 0) {
#pragma unroll
    for (int m = 0; m < MT; m++) {
      out[27 * TM * TN + 16 * m + g] = bias_sum[m][0];
      out[27 * TM * TN + 16 * m + g + 8] = bias_sum[m][1];
    }
  }
}

// The blocks' sums, in a fixed order: 32 outputs and 8 groups of blocks per
// thread block. g32: the first three rows are one channel's.
__global__ void __launch_bounds__(256) k_wgrad_fold(const float *__restrict__ partial, int blocks,
    int tm, int tn, int parts_n, int co, int ci, int g32, float *__restrict__ dw,
    float *__restrict__ db)
{
  __shared__ float sm[8][32];
  const int lane = threadIdx.x & 31, grp = threadIdx.x >> 5;
  const int nw = 27 * co * ci, i = blockIdx.x * 32 + lane;
  const int stride = 27 * tm * tn + tm;
  float s = 0.0f;
  if (i < nw + co) {
    int part, at, step;  // step: to the next row of one channel
    if (i < nw) {
      const int n = i % ci, m = (i / ci) % co, tap = i / (ci * co);
      part = (m / tm) * parts_n + n / tn;
      at = (tap * tm + m % tm) * tn + n % tn;
      step = tn;
    } else {
      const int m = i - nw;
      part = (m / tm) * parts_n;
      at = 27 * tm * tn + m % tm;
      step = 1;
    }
    const float *p = partial + (int64_t)part * blocks * stride + at;
    for (int b = grp; b < blocks; b += 8) {
      const float *q = p + (int64_t)b * stride;
      s += g32 ? (q[2 * step] + q[step]) + q[0] : q[0];
    }
  }
  sm[grp][lane] = s;
  __syncthreads();
  if (grp == 0 && i < nw + co) {
    float v = 0.0f;
#pragma unroll
    for (int q = 0; q < 8; q++) v += sm[q][lane];
    if (i < nw) dw[i] = v;
    else db[i - nw] = v;
  }
}

struct Plan {
  int tm, tn, parts, parts_n, run, xt, yc, yt, items, blocks, chain;
};

// Tiles of 16 x 16, 16 x 48, 32 x 16 or 32 x 32 channels (the accumulators of
// three taps fit the registers); marches short enough that every block of two
// per SM has one, long enough that the two rows around a march do not count
Plan plan(int co, int ci, int B, int Z, int Y, int X)
{
  Plan p;
  p.tm = co <= 16 ? 16 : 32;
  p.tn = p.tm == 16 ? (ci == 48 ? 48 : 16) : (ci == 16 ? 16 : 32);
  p.parts_n = ci <= p.tn ? 1 : ci / p.tn;
  p.parts = (co <= p.tm ? 1 : co / p.tm) * p.parts_n;
  const int up16 = (X + 15) / 16 * 16;
  p.run = up16 < kRun ? up16 : kRun;
  p.xt = (X + p.run - 1) / p.run;
  const int wave = kWave / p.parts;
  const int64_t columns = (int64_t)B * Z * p.xt;
  p.yc = Y;
  while (p.yc > 8 && columns * ((Y + p.yc - 1) / p.yc) < 2 * wave) p.yc = (p.yc + 1) / 2;
  p.yt = (Y + p.yc - 1) / p.yc;
  p.items = (int)(columns * p.yt);
  p.blocks = p.items < wave ? p.items : wave;
  const int64_t chain = ((int64_t)B * Z * Y * X + 255) / 256;
  p.chain = chain < 512 ? 512 : (int)chain;
  return p;
}

template <int TM, int TN, bool G32, bool ROWS>
bool launch(const Plan &p, const Args &a)
{
  constexpr int bytes = Layout<TM, TN>::kSmem;
  static bool set[64] = {};
  int dev = 0;
  if (!cuda_ok(cudaGetDevice(&dev), "cudaGetDevice")) return false;
  if (dev >= 0 && dev < 64 && !set[dev]) {
    if (!cuda_ok(cudaFuncSetAttribute(k_wgrad<TM, TN, G32, ROWS>,
                     cudaFuncAttributeMaxDynamicSharedMemorySize, bytes),
            "k_wgrad shared memory"))
      return false;
    set[dev] = true;
  }
  k_wgrad<TM, TN, G32, ROWS><<<dim3(p.blocks, p.parts), kThreads, bytes, stream()>>>(a);
  return launched("k_wgrad");
}

}  // namespace

int64_t wgrad_scratch(int co, int ci, int B, int Z, int Y, int X)
{
  const Plan p = plan(co, ci, B, Z, Y, X);
  return (int64_t)p.parts * p.blocks * (27 * p.tm * p.tn + p.tm);
}

bool wgrad_conv(const WgradSrc &s0, const WgradSrc &s1, const void *g, const float *g32, int co,
    int ci, int B, int Z, int Y, int X, float *scratch, float *dw, float *db)
{
  const Plan p = plan(co, ci, B, Z, Y, X);
  Args a;
  a.s0 = s0;
  a.s1 = s1;
  a.g = static_cast<const bf16 *>(g);
  a.g32 = g32;
  a.B = B;
  a.Z = Z;
  a.Y = Y;
  a.X = X;
  a.run = p.run;
  a.xt = p.xt;
  a.yc = p.yc;
  a.yt = p.yt;
  a.items = p.items;
  a.co = co;
  a.parts_n = p.parts_n;
  a.chain = p.chain;
  a.partial = scratch;
  bool ok = false;
  if (g32) ok = launch<16, 16, true, true>(p, a);
  else if (ci < 16) ok = launch<16, 16, false, true>(p, a);
  else if (p.tm == 16 && p.tn == 16) ok = launch<16, 16, false, false>(p, a);
  else if (p.tm == 16 && p.tn == 48) ok = launch<16, 48, false, false>(p, a);
  else if (p.tm == 32 && p.tn == 16) ok = launch<32, 16, false, false>(p, a);
  else ok = launch<32, 32, false, false>(p, a);
  if (!ok) return false;
  const int n = 27 * co * ci + co;
  k_wgrad_fold<<<(n + 31) / 32, 256, 0, stream()>>>(scratch, p.blocks, p.tm, p.tn, p.parts_n, co, ci,
      g32 ? 1 : 0, dw, db);
  return launched("k_wgrad_fold");
}

}  // namespace nusif
