// Learned pressure warm start: a 3-level 3D U-Net trained and run on the GPU
// with this file's kernels (no reference counterpart: the reference solver has
// no learned component).
//
// Network (volumes channels-last [B][Z][Y][X][C]; every conv 3x3x3 with zero
// padding; weights W[tap][cout][cin], tap = 9(dz+1) + 3(dy+1) + (dx+1)):
//   e0a 2->16, e0b 16->16 | pool | e1a 16->32, e1b 32->32 | pool | e2a 32->64
//   | up, concat [up(e2a), e1b] | d1a 96->32, d1b 32->32 | up, concat
//   [up(d1b), e0b] | d0a 48->16, d0b 16->16 | out 16->1 (linear, FP32).
// ReLU after every conv but the last; pool = 2x2x2 mean, up = nearest.
//
// Precision: BF16 weights and activations, FP32 accumulation (tensor cores),
// FP32 master weights, gradients and Adam state. A layer's output gradient
// times its ReLU mask is rounded to BF16 before the tensor-core kernels use it.
//
// Kernels:
//  - k_conv_col, k_conv_tc (unet_tc.cu): the forward and input-gradient
//    convolutions on the 5th-generation tensor cores (tcgen05.mma, TMEM
//    accumulators, TMA staging) whenever the volume's rows tile into 128-cell
//    blocks, marching over planes for layers of up to 48 channels; the
//    96-channel layer's upsampled source is then materialised by k_upsample.
//  - k_conv_mma: implicit-GEMM conv on the tensor cores (mma.sync m16n8k16
//    BF16 -> FP32): M = cells (16 per warp), N = output channels, K = 27 taps x
//    input channels in chunks of 16. Its loader reads up to two sources, the
//    first optionally at half resolution (nearest upsampling and the concat
//    of the decoder are never materialised). The same kernel computes input
//    gradients with tap-flipped, transposed weights.
//  - k_wgrad (unet_wgrad.cu): weight gradients of every layer as GEMMs over
//    the cells on the tensor cores.
//  - plain FP32 kernels for the 2-channel input layer and the 1-channel output
//    layer, pooling, masks, the loss and Adam.
#include <cuda_bf16.h>

#include <cmath>
#include <cstdint>
#include <cstring>
#include <utility>
#include <vector>

#include "nusif_internal.h"
#include "unet_internal.h"
#include "unet_tc.h"
#include "unet_wgrad.h"

namespace nusif {
namespace {

using bf16 = __nv_bfloat16;

constexpr int kLayers = 10;
enum { L_E0A, L_E0B, L_E1A, L_E1B, L_E2A, L_D1A, L_D1B, L_D0A, L_D0B, L_OUT };
struct LayerDesc {
  int cin, cout;
};
constexpr LayerDesc kDesc[kLayers] = { { 2, 16 }, { 16, 16 }, { 16, 32 }, { 32, 32 }, { 32, 64 },
  { 96, 32 }, { 32, 32 }, { 48, 16 }, { 16, 16 }, { 16, 1 } };

// ------------------------------------------------------------------ device helpers

__device__ __forceinline__ uint32_t ld_pair(const bf16 *p)
{
  return *reinterpret_cast<const uint32_t *>(p);
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi)
{
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t *>(&v);
}

// D += A(16x16, row) * B(16x8, col), BF16 inputs, FP32 accumulators
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0,
    uint32_t b1)
{
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
      "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

struct Vol {
  int B, Z, Y, X;
  __host__ __device__ int64_t cells() const { return (int64_t)B * Z * Y * X; }
};

__device__ __forceinline__ void decompose(const Vol &v, int64_t c, int &b, int &z, int &y, int &x)
{
  x = (int)(c % v.X);
  int64_t r = c / v.X;
  y = (int)(r % v.Y);
  r /= v.Y;
  z = (int)(r % v.Z);
  b = (int)(r / v.Z);
}

// ------------------------------------------------------------------ tensor-core conv

struct ConvSrc {
  const bf16 *p;
  int c;   // channels (multiple of 16)
  int up;  // 1: stored at half resolution, read by nearest upsampling
};

struct ConvArgs {
  ConvSrc s0, s1;   // s1.c == 0: one source
  Vol v;            // output (= full input) resolution
  const bf16 *w;    // [27][COUT][cin]
  const float *bias;
  int relu;
  void *out;        // bf16 or float [cells][COUT]
};

// One warp = 16 consecutive output cells x all COUT channels. Rows g and g+8
// of the mma fragments are this thread's two cells. A step is a tap and 16
// input channels; the fragments of the next D - 1 steps are in flight while one
// is multiplied (they come straight from L1 and L2, whose latency is what a
// warp waits for). Same products in the same order whatever D. Per call, 4 x 60 x
// 12 x 12 cells: 32 channels out 29 -> 21 us (D = 6: 36), 16 channels 24 -> 21; 4 x 64
// x 60 x 60: 16 channels 408 -> 375 us (D = 4: 425).
template <int COUT, bool OUT_BF16>
__global__ void __launch_bounds__(128) k_conv_mma(ConvArgs a)
{
  constexpr int D = COUT <= 16 ? 2 : COUT <= 32 ? 4 : COUT <= 48 ? 3 : 2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int64_t ncell = a.v.cells();
  const int64_t base = ((int64_t)blockIdx.x * 4 + warp) * 16;
  if (base >= ncell) return;
  const int cin = a.s0.c + a.s1.c;
  int cb[2], cz[2], cy[2], cx[2];
  bool live[2];
  for (int r = 0; r < 2; r++) {
    const int64_t c = base + g + 8 * r;
    live[r] = c < ncell;
    decompose(a.v, live[r] ? c : 0, cb[r], cz[r], cy[r], cx[r]);
  }
  const int hZ = a.v.Z >> 1, hY = a.v.Y >> 1, hX = a.v.X >> 1;
  float acc[COUT / 8][4];
#pragma unroll
  for (int j = 0; j < COUT / 8; j++) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0f;
  struct Step {
    uint32_t A[4], W[COUT / 8][2];
  };
  // the next step to load: tap (dz, dy, dx) and channel, and the tap's cells
  int tap = -1, kc = cin;
  bool ok[2];
  int64_t n1[2], n0[2];
  const auto load = [&](Step &q) {
    if (kc == cin) {
      kc = 0;
      if (++tap == 27) return;
      const int dz = tap / 9 - 1, dy = (tap / 3) % 3 - 1, dx = tap % 3 - 1;
#pragma unroll
      for (int r = 0; r < 2; r++) {
        const int z = cz[r] + dz, y = cy[r] + dy, x = cx[r] + dx;
        ok[r] = live[r] && z >= 0 && z < a.v.Z && y >= 0 && y < a.v.Y && x >= 0 && x < a.v.X;
        n1[r] = ok[r] ? (((int64_t)cb[r] * a.v.Z + z) * a.v.Y + y) * a.v.X + x : 0;
        n0[r] = !a.s0.up ? n1[r]
                         : (ok[r] ? (((int64_t)cb[r] * hZ + (z >> 1)) * hY + (y >> 1)) * hX + (x >> 1)
                                  : 0);
      }
    }
    const bool first = kc < a.s0.c;
    const bf16 *src = first ? a.s0.p : a.s1.p;
    const int cs = first ? a.s0.c : a.s1.c;
    const int c0 = (first ? kc : kc - a.s0.c) + 2 * t;
    const int64_t o0 = (first ? n0[0] : n1[0]) * cs + c0;
    const int64_t o1 = (first ? n0[1] : n1[1]) * cs + c0;
    q.A[0] = ok[0] ? ld_pair(src + o0) : 0u;
    q.A[1] = ok[1] ? ld_pair(src + o1) : 0u;
    q.A[2] = ok[0] ? ld_pair(src + o0 + 8) : 0u;
    q.A[3] = ok[1] ? ld_pair(src + o1 + 8) : 0u;
    const bf16 *wr = a.w + ((int64_t)tap * COUT + g) * cin + kc + 2 * t;
#pragma unroll
    for (int j = 0; j < COUT / 8; j++, wr += 8 * cin) {
      q.W[j][0] = __ldg(reinterpret_cast<const unsigned *>(wr));
      q.W[j][1] = __ldg(reinterpret_cast<const unsigned *>(wr + 8));
    }
    kc += 16;
  };
  Step f[D];
#pragma unroll
  for (int u = 0; u < D - 1; u++) load(f[u]);  // at least 27 steps
  const int steps = 27 * (cin / 16);
  for (int s = 0; s < steps; s += D) {
#pragma unroll
    for (int u = 0; u < D; u++) {
      if (s + u >= steps) break;
      if (s + u + D - 1 < steps) load(f[(u + D - 1) % D]);
#pragma unroll
      for (int j = 0; j < COUT / 8; j++) mma_bf16(acc[j], f[u].A, f[u].W[j][0], f[u].W[j][1]);
    }
  }
#pragma unroll
  for (int r = 0; r < 2; r++) {
    if (!live[r]) continue;
    const int64_t c = base + g + 8 * r;
#pragma unroll
    for (int j = 0; j < COUT / 8; j++) {
      const int co = 8 * j + 2 * t;
      float v0 = acc[j][2 * r], v1 = acc[j][2 * r + 1];
      if (a.bias) {
        v0 += a.bias[co];
        v1 += a.bias[co + 1];
      }
      if (a.relu) {
        v0 = fmaxf(v0, 0.0f);
        v1 = fmaxf(v1, 0.0f);
      }
      if (OUT_BF16)
        *reinterpret_cast<uint32_t *>(static_cast<bf16 *>(a.out) + c * COUT + co) = pack_bf16(v0, v1);
      else
        *reinterpret_cast<float2 *>(static_cast<float *>(a.out) + c * COUT + co) = make_float2(v0, v1);
    }
  }
}

// ------------------------------------------------------------------ plain layers

// e0a: 2 -> 16, ReLU (FP32 arithmetic on BF16 values)
__global__ void __launch_bounds__(256) k_conv_first(const bf16 *__restrict__ x, Vol v,
    const bf16 *__restrict__ w, const float *__restrict__ bias, bf16 *__restrict__ y)
{
  __shared__ float ws[27 * 16 * 2];
  for (int i = threadIdx.x; i < 27 * 32; i += blockDim.x) ws[i] = __bfloat162float(w[i]);
  __syncthreads();
  const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c >= v.cells()) return;
  int b, z, yy, xx;
  decompose(v, c, b, z, yy, xx);
  float acc[16];
#pragma unroll
  for (int o = 0; o < 16; o++) acc[o] = bias[o];
  for (int tap = 0; tap < 27; tap++) {
    const int nz = z + tap / 9 - 1, ny = yy + (tap / 3) % 3 - 1, nx = xx + tap % 3 - 1;
    if (nz < 0 || nz >= v.Z || ny < 0 || ny >= v.Y || nx < 0 || nx >= v.X) continue;
    const int64_t n = (((int64_t)b * v.Z + nz) * v.Y + ny) * v.X + nx;
    const float x0 = __bfloat162float(x[2 * n]), x1 = __bfloat162float(x[2 * n + 1]);
#pragma unroll
    for (int o = 0; o < 16; o++) acc[o] += ws[(tap * 16 + o) * 2] * x0 + ws[(tap * 16 + o) * 2 + 1] * x1;
  }
#pragma unroll
  for (int o = 0; o < 16; o += 2)
    *reinterpret_cast<uint32_t *>(y + c * 16 + o) =
        pack_bf16(fmaxf(acc[o], 0.0f), fmaxf(acc[o + 1], 0.0f));
}

// out: 16 -> 1, linear, FP32 output
__global__ void __launch_bounds__(256) k_conv_last(const bf16 *__restrict__ x, Vol v,
    const bf16 *__restrict__ w, const float *__restrict__ bias, float *__restrict__ y)
{
  __shared__ float ws[27 * 16];
  for (int i = threadIdx.x; i < 27 * 16; i += blockDim.x) ws[i] = __bfloat162float(w[i]);
  __syncthreads();
  const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c >= v.cells()) return;
  int b, z, yy, xx;
  decompose(v, c, b, z, yy, xx);
  float acc = bias[0];
  for (int tap = 0; tap < 27; tap++) {
    const int nz = z + tap / 9 - 1, ny = yy + (tap / 3) % 3 - 1, nx = xx + tap % 3 - 1;
    if (nz < 0 || nz >= v.Z || ny < 0 || ny >= v.Y || nx < 0 || nx >= v.X) continue;
    const bf16 *xn = x + ((((int64_t)b * v.Z + nz) * v.Y + ny) * v.X + nx) * 16;
#pragma unroll
    for (int i = 0; i < 16; i++) acc += ws[tap * 16 + i] * __bfloat162float(xn[i]);
  }
  y[c] = acc;
}

// masked input gradient of the output layer: G[c][i] = (sum over taps of
// dout[c - off] W[tap][i]) where y > 0, in BF16; four cells of a row per
// thread, so a tap's weights are read once for four
__global__ void __launch_bounds__(128) k_conv_last_dgrad(const float *__restrict__ dout, Vol v,
    const bf16 *__restrict__ w, const bf16 *__restrict__ y, bf16 *__restrict__ g)
{
  __shared__ __align__(16) float ws[27 * 16];
  for (int i = threadIdx.x; i < 27 * 16; i += blockDim.x) ws[i] = __bfloat162float(w[i]);
  __syncthreads();
  const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (4 * q >= v.cells()) return;
  int b, z, yy, x0;
  decompose(v, 4 * q, b, z, yy, x0);  // x is a multiple of 4
  float acc[4][16];
#pragma unroll
  for (int c = 0; c < 4; c++)
#pragma unroll
    for (int i = 0; i < 16; i++) acc[c][i] = 0.0f;
  for (int zy = 0; zy < 9; zy++) {
    const int nz = z - (zy / 3 - 1), ny = yy - (zy % 3 - 1);
    if (nz < 0 || nz >= v.Z || ny < 0 || ny >= v.Y) continue;
    const float *row = dout + (((int64_t)b * v.Z + nz) * v.Y + ny) * v.X + x0;
    const float4 m = *reinterpret_cast<const float4 *>(row);
    const float d[6] = { x0 > 0 ? row[-1] : 0.0f, m.x, m.y, m.z, m.w,
                         x0 + 4 < v.X ? row[4] : 0.0f };
#pragma unroll
    for (int dx = 0; dx < 3; dx++) {  // tap dx - 1 reads the cell at x - (dx - 1)
      const float *wt = ws + (3 * zy + dx) * 16;
#pragma unroll
      for (int i = 0; i < 16; i++)
#pragma unroll
        for (int c = 0; c < 4; c++) acc[c][i] += d[c + 2 - dx] * wt[i];
    }
  }
#pragma unroll
  for (int c = 0; c < 4; c++) {
    const uint4 *k = reinterpret_cast<const uint4 *>(y + (4 * q + c) * 16);
    uint4 *o = reinterpret_cast<uint4 *>(g + (4 * q + c) * 16);
#pragma unroll
    for (int h = 0; h < 2; h++) {
      float t[8], m[8];
      const uint4 yv = k[h];
      const uint32_t u[4] = { yv.x, yv.y, yv.z, yv.w };
#pragma unroll
      for (int e = 0; e < 8; e++) {
        m[e] = __uint_as_float(e & 1 ? u[e / 2] & 0xffff0000u : u[e / 2] << 16);
        t[e] = m[e] > 0.0f ? acc[c][8 * h + e] : 0.0f;
      }
      o[h] = make_uint4(pack_bf16(t[0], t[1]), pack_bf16(t[2], t[3]), pack_bf16(t[4], t[5]),
          pack_bf16(t[6], t[7]));
    }
  }
}

// ------------------------------------------------------------------ elementwise

// the 2-channel FP32 input as BF16, once as [cells][2] (the plain first
// layer) and once zero-padded to [cells][16] (the tensor-core first layer and
// its weight gradient: channels in groups of 16)
__global__ void k_input_bf16(const float *__restrict__ x, int64_t n, bf16 *__restrict__ x2,
    bf16 *__restrict__ x16)
{
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n;
       c += (int64_t)gridDim.x * blockDim.x) {
    const float2 a = reinterpret_cast<const float2 *>(x)[c];
    const uint32_t v = pack_bf16(a.x, a.y);
    reinterpret_cast<uint32_t *>(x2)[c] = v;
    uint4 *o = reinterpret_cast<uint4 *>(x16 + c * 16);
    o[0] = make_uint4(v, 0u, 0u, 0u);
    o[1] = make_uint4(0u, 0u, 0u, 0u);
  }
}

// W[27][co][ci] (FP32) -> BF16 [27][16][16], zero outside co x ci (the first
// and last layers on the tensor cores)
__global__ void k_pad_weights16(const float *__restrict__ w, int co, int ci, bf16 *__restrict__ wp)
{
  const int n = 27 * 16 * 16;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int tap = i / 256, o = (i / 16) % 16, k = i % 16;
    wp[i] = __float2bfloat16_rn(o < co && k < ci ? w[(tap * co + o) * ci + k] : 0.0f);
  }
}

// nearest upsampling of a [half cells][C] BF16 volume to full resolution, 8
// channels (16 bytes) per thread
__global__ void k_upsample(const bf16 *__restrict__ c, Vol fv, int C, bf16 *__restrict__ f)
{
  const int g8 = C / 8;
  const int64_t n = fv.cells() * g8;
  const int hZ = fv.Z / 2, hY = fv.Y / 2, hX = fv.X / 2;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int grp = (int)(i % g8);
    int b, z, y, x;
    decompose(fv, i / g8, b, z, y, x);
    const int64_t cc = (((int64_t)b * hZ + (z >> 1)) * hY + (y >> 1)) * hX + (x >> 1);
    reinterpret_cast<uint4 *>(f)[i] = reinterpret_cast<const uint4 *>(c)[cc * g8 + grp];
  }
}

// One thread per 8 channels of a cell in the kernels below: threads run over
// the 8-channel groups of a row of cells, blocks over rows and planes (no
// division of a flat index). groups: of a row.
struct RowIndex {
  int g, y;  // group in the row, row
  int64_t zb, zstep;
};

__device__ __forceinline__ RowIndex row_index()
{
  return { (int)(blockIdx.x * blockDim.x + threadIdx.x), (int)blockIdx.y, (int64_t)blockIdx.z,
    (int64_t)gridDim.z };
}

__device__ __forceinline__ void unpack8(uint4 w, float (&f)[8])
{
  const uint32_t u[4] = { w.x, w.y, w.z, w.w };
#pragma unroll
  for (int e = 0; e < 8; e++)  // BF16 is the upper half of a float
    f[e] = __uint_as_float(e & 1 ? u[e / 2] & 0xffff0000u : u[e / 2] << 16);
}

__device__ __forceinline__ uint4 pack8(const float (&f)[8])
{
  return make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]),
      pack_bf16(f[6], f[7]));
}

__device__ __forceinline__ void load8(const float *p, float (&f)[8])
{
  const float4 a = reinterpret_cast<const float4 *>(p)[0], b = reinterpret_cast<const float4 *>(p)[1];
  f[0] = a.x;
  f[1] = a.y;
  f[2] = a.z;
  f[3] = a.w;
  f[4] = b.x;
  f[5] = b.y;
  f[6] = b.z;
  f[7] = b.w;
}

// bf16(d * (Y > 0)) of 8 channels
__device__ __forceinline__ uint4 masked8(const float (&d)[8], uint4 y)
{
  float m[8], r[8];
  unpack8(y, m);
#pragma unroll
  for (int e = 0; e < 8; e++) r[e] = m[e] > 0.0f ? d[e] : 0.0f;
  return pack8(r);
}

// G = bf16(dY * (Y > 0)), n groups of 8
__global__ void k_relu_mask(const float *__restrict__ dy, const bf16 *__restrict__ y, int64_t n,
    bf16 *__restrict__ g)
{
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    float d[8];
    load8(dy + 8 * i, d);
    reinterpret_cast<uint4 *>(g)[i] = masked8(d, reinterpret_cast<const uint4 *>(y)[i]);
  }
}

// 2x2x2 mean of a [fine cells][C] BF16 volume (grid over the coarse volume)
__global__ void k_pool(const bf16 *__restrict__ f, Vol cv, int C, bf16 *__restrict__ o)
{
  const int g8 = C / 8;
  const RowIndex r = row_index();
  if (r.g >= cv.X * g8) return;
  const int x = r.g / g8, grp = r.g - x * g8;
  for (int64_t zb = r.zb; zb < (int64_t)cv.B * cv.Z; zb += r.zstep) {
    float s[8];
#pragma unroll
    for (int e = 0; e < 8; e++) s[e] = 0.0f;
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const int64_t fc =
          ((2 * zb + (q >> 2)) * (2 * cv.Y) + 2 * r.y + ((q >> 1) & 1)) * (2 * cv.X) + 2 * x + (q & 1);
      float v[8];
      unpack8(reinterpret_cast<const uint4 *>(f)[fc * g8 + grp], v);
#pragma unroll
      for (int e = 0; e < 8; e++) s[e] += v[e];
    }
#pragma unroll
    for (int e = 0; e < 8; e++) s[e] *= 0.125f;
    reinterpret_cast<uint4 *>(o)[((zb * cv.Y + r.y) * cv.X + x) * g8 + grp] = pack8(s);
  }
}

// the masked gradient of a layer whose output went to the next layer's skip
// (gf, fine) and to the mean pool (gc, coarse: a child's share is an eighth)
__global__ void k_pool_back_mask(const float *__restrict__ gf, const float *__restrict__ gc, Vol fv,
    int C, const bf16 *__restrict__ y, bf16 *__restrict__ g)
{
  const int g8 = C / 8;
  const RowIndex r = row_index();
  if (r.g >= fv.X * g8) return;
  const int x = r.g / g8, grp = r.g - x * g8;
  for (int64_t zb = r.zb; zb < (int64_t)fv.B * fv.Z; zb += r.zstep) {  // Z is even: (b, z / 2) is zb / 2
    const int64_t i = ((zb * fv.Y + r.y) * fv.X + x) * g8 + grp;
    const int64_t c = (((zb >> 1) * (fv.Y / 2) + (r.y >> 1)) * (fv.X / 2) + (x >> 1)) * g8 + grp;
    float a[8], b[8];
    load8(gf + 8 * i, a);
    load8(gc + 8 * c, b);
#pragma unroll
    for (int e = 0; e < 8; e++) a[e] += 0.125f * b[e];
    reinterpret_cast<uint4 *>(g)[i] = masked8(a, reinterpret_cast<const uint4 *>(y)[i]);
  }
}

// the masked gradient of a layer whose output was upsampled: the sum over a
// coarse cell's 8 children of the first Cu channels of a fine gradient of
// `stride` channels (grid over the coarse volume)
__global__ void k_up_back_mask(const float *__restrict__ d, int stride, Vol cv, int Cu,
    const bf16 *__restrict__ y, bf16 *__restrict__ g)
{
  const int g8 = Cu / 8;
  const RowIndex r = row_index();
  if (r.g >= cv.X * g8) return;
  const int x = r.g / g8, grp = r.g - x * g8;
  for (int64_t zb = r.zb; zb < (int64_t)cv.B * cv.Z; zb += r.zstep) {
    float s[8];
#pragma unroll
    for (int e = 0; e < 8; e++) s[e] = 0.0f;
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const int64_t fc =
          ((2 * zb + (q >> 2)) * (2 * cv.Y) + 2 * r.y + ((q >> 1) & 1)) * (2 * cv.X) + 2 * x + (q & 1);
      float v[8];
      load8(d + fc * stride + 8 * grp, v);
#pragma unroll
      for (int e = 0; e < 8; e++) s[e] += v[e];
    }
    const int64_t i = ((zb * cv.Y + r.y) * cv.X + x) * g8 + grp;
    reinterpret_cast<uint4 *>(g)[i] = masked8(s, reinterpret_cast<const uint4 *>(y)[i]);
  }
}

// the last Cs channels of a gradient of Cu + Cs channels, n groups of 8
__global__ void k_skip_part(const float *__restrict__ dcat, int64_t n, int Cu, int Cs,
    float *__restrict__ dskip)
{
  const int g8 = Cs / 8;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = i / g8;
    const float4 *s =
        reinterpret_cast<const float4 *>(dcat + c * (Cu + Cs) + Cu + 8 * (i - c * g8));
    reinterpret_cast<float4 *>(dskip)[2 * i] = s[0];
    reinterpret_cast<float4 *>(dskip)[2 * i + 1] = s[1];
  }
}

// squared error partial sums and the loss gradient 2 (out - t) / n
__global__ void __launch_bounds__(256) k_mse(const float *__restrict__ out,
    const float *__restrict__ tgt, int64_t n, int64_t chunk, float *__restrict__ dout,
    double *__restrict__ partial)
{
  __shared__ double sm[256];
  const int64_t c_begin = blockIdx.x * chunk, c_end = min(c_begin + chunk, n);
  const float inv = 2.0f / (float)n;
  double s = 0.0;
  for (int64_t i = c_begin + threadIdx.x; i < c_end; i += 256) {
    const float d = out[i] - tgt[i];
    s += (double)d * d;
    if (dout) dout[i] = inv * d;
  }
  sm[threadIdx.x] = s;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) sm[threadIdx.x] += sm[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = sm[0];
}

__global__ void __launch_bounds__(256) k_fold_loss(const double *__restrict__ partial, int nb,
    int64_t n, float *loss)
{
  __shared__ double sm[256];
  double s = 0.0;
  for (int i = threadIdx.x; i < nb; i += 256) s += partial[i];
  sm[threadIdx.x] = s;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) sm[threadIdx.x] += sm[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) *loss = (float)(sm[0] / (double)n);
}

__global__ void k_adam(float *__restrict__ w, const float *__restrict__ g, float *__restrict__ m,
    float *__restrict__ v, int64_t n, float lr, float b1, float b2, float eps, float c1, float c2)
{
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    w[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  }
}

// BF16 copies of one layer's weights: W[tap][co][ci] and, for input gradients,
// the tap-flipped transpose Wt[tap][ci][co] = W[26 - tap][co][ci]
__global__ void k_layer_bf16(const float *__restrict__ w, int co, int ci, bf16 *__restrict__ wb,
    bf16 *__restrict__ wt)
{
  const int n = 27 * co * ci;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    wb[i] = __float2bfloat16_rn(w[i]);
    if (wt) {
      const int tap = i / (co * ci), r = i % (co * ci), o = r / ci, k = r % ci;
      wt[((26 - tap) * ci + k) * co + o] = __float2bfloat16_rn(w[i]);
    }
  }
}

int blocks_for(int64_t n, int threads = 256)
{
  int64_t b = (n + threads - 1) / threads;
  if (b > 152 * 32) b = 152 * 32;
  return (int)(b < 1 ? 1 : b);
}

}  // namespace

// ------------------------------------------------------------------ host side

struct UNetState {
  int64_t w_off[kLayers], b_off[kLayers];
  int64_t nparam = 0;
  float *master = nullptr, *grad = nullptr, *m = nullptr, *v = nullptr;  // device FP32
  bf16 *wb[kLayers] = {}, *wt[kLayers] = {};
  int adam_t = 0;
  // workspace for the current volume
  Vol vol = { 0, 0, 0, 0 };
  int64_t cap0 = 0;  // level-0 cells the workspace holds
  bf16 *x = nullptr, *e0a = nullptr, *e0b = nullptr, *p0 = nullptr, *e1a = nullptr,
       *e1b = nullptr, *p1 = nullptr, *e2a = nullptr, *d1a = nullptr, *d1b = nullptr,
       *d0a = nullptr, *d0b = nullptr, *G = nullptr,
       *G2 = nullptr;  // masked output gradient of the current layer, and of the next
  float *out = nullptr, *dout = nullptr, *F1 = nullptr, *F2 = nullptr, *Fe0b = nullptr,
        *Fe1b = nullptr, *partial = nullptr;
  int64_t partial_cap = 0;
  bf16 *up1 = nullptr;                  // materialised up(e2a) [n1][64]
  bf16 *x16 = nullptr;                  // input zero-padded to 16 channels
  bf16 *w_first16 = nullptr, *w_last16 = nullptr;  // e0a and out weights padded to [27][16][16]
  int *err = nullptr;                   // device: a tensor-core kernel's wait timed out
  int use_tc = 1;                       // tcgen05 kernels where the volume allows
  double *loss_partial = nullptr;
  float *loss = nullptr;  // device scalar
  std::vector<void *> ws;
};

namespace {

template <typename T>
bool dalloc(UNetState *u, T **p, int64_t n)
{
  if (!cuda_ok(cudaMalloc(reinterpret_cast<void **>(p), (size_t)n * sizeof(T)), "cudaMalloc(unet)"))
    return false;
  u->ws.push_back(*p);
  return true;
}

void free_workspace(UNetState *u)
{
  for (void *p : u->ws) cudaFree(p);
  u->ws.clear();
  u->cap0 = 0;
}

bool ensure_workspace(UNetState *u, const Vol &v)
{
  if (v.Z % 4 || v.Y % 4 || v.X % 4 || v.B < 1 || v.Z < 4 || v.Y < 4 || v.X < 4) {
    fail(NUSIF_ERR_ARG, "unet: volume %dx%dx%d (batch %d) needs every edge a multiple of 4", v.X,
        v.Y, v.Z, v.B);
    return false;
  }
  u->vol = v;
  const int64_t n0 = v.cells();
  if (n0 <= u->cap0) return true;
  cudaStreamSynchronize(stream());
  free_workspace(u);
  const int64_t n1 = n0 / 8, n2 = n0 / 64;
  bool ok = dalloc(u, &u->x, 2 * n0) && dalloc(u, &u->e0a, 16 * n0) && dalloc(u, &u->e0b, 16 * n0) &&
            dalloc(u, &u->p0, 16 * n1) && dalloc(u, &u->e1a, 32 * n1) && dalloc(u, &u->e1b, 32 * n1) &&
            dalloc(u, &u->p1, 32 * n2) && dalloc(u, &u->e2a, 64 * n2) && dalloc(u, &u->d1a, 32 * n1) &&
            dalloc(u, &u->d1b, 32 * n1) && dalloc(u, &u->d0a, 16 * n0) && dalloc(u, &u->d0b, 16 * n0) &&
            dalloc(u, &u->G, 16 * n0) && dalloc(u, &u->G2, 16 * n0) && dalloc(u, &u->out, n0) && dalloc(u, &u->dout, n0) &&
            dalloc(u, &u->F1, 48 * n0) && dalloc(u, &u->F2, 16 * n0) && dalloc(u, &u->Fe0b, 16 * n0) &&
            dalloc(u, &u->Fe1b, 32 * n1) && dalloc(u, &u->loss_partial, 1024) &&
            dalloc(u, &u->up1, 64 * n1) &&
            dalloc(u, &u->x16, 16 * n0);
  if (!ok) return false;
  u->cap0 = n0;
  return true;
}

bool ensure_partial(UNetState *u, int64_t n)
{
  if (n <= u->partial_cap) return true;
  cudaStreamSynchronize(stream());
  if (u->partial) cudaFree(u->partial);
  u->partial = nullptr;
  u->partial_cap = 0;
  if (!cuda_ok(cudaMalloc(&u->partial, (size_t)n * sizeof(float)), "cudaMalloc(unet partial)"))
    return false;
  u->partial_cap = n;
  return true;
}

template <int COUT, bool OUT_BF16>
bool conv_mma(const ConvSrc &s0, const ConvSrc &s1, const Vol &v, const bf16 *w, const float *bias,
    int relu, void *out)
{
  ConvArgs a;
  a.s0 = s0;
  a.s1 = s1;
  a.v = v;
  a.w = w;
  a.bias = bias;
  a.relu = relu;
  a.out = out;
  const int64_t warps = (v.cells() + 15) / 16;
  k_conv_mma<COUT, OUT_BF16><<<(unsigned)((warps + 3) / 4), 128, 0, stream()>>>(a);
  return launched("k_conv_mma");
}

bool tc_ok(const UNetState *u, const Vol &v, int n, int c0, int c1)
{
  return u->use_tc && tc_conv_supported(v.X, v.Y, v.Z, v.B, n, c0, c1);
}

// forward conv of a tensor-core layer (BF16 out, bias, ReLU)
bool fwd(UNetState *u, int l, const ConvSrc &s0, const ConvSrc &s1, const Vol &v, bf16 *out)
{
  const float *bias = u->master + u->b_off[l];
  if (tc_ok(u, v, kDesc[l].cout, s0.c, s1.c)) {
    const bf16 *a0 = s0.p;
    int up = s0.up;
    if (up && !tc_conv_marches(kDesc[l].cout, s0.c + s1.c)) {
      // the decoder's upsampled source, materialised at full resolution
      k_upsample<<<blocks_for(v.cells() * (s0.c / 8)), 256, 0, stream()>>>(s0.p, v, s0.c, u->up1);
      if (!launched("k_upsample")) return false;
      a0 = u->up1;
      up = 0;
    }
    return tc_conv(a0, s0.c, s1.p, s1.c, v.B, v.Z, v.Y, v.X, u->wb[l], kDesc[l].cout, bias, 1,
        TC_BF16, out, u->err, up);
  }
  switch (kDesc[l].cout) {
  case 16: return conv_mma<16, true>(s0, s1, v, u->wb[l], bias, 1, out);
  case 32: return conv_mma<32, true>(s0, s1, v, u->wb[l], bias, 1, out);
  case 64: return conv_mma<64, true>(s0, s1, v, u->wb[l], bias, 1, out);
  }
  fail(NUSIF_ERR_STATE, "unet: no forward kernel for %d output channels", kDesc[l].cout);
  return false;
}

// input gradient of a tensor-core layer: G (cout channels) -> FP32 [cells][cin]
bool dgrad(UNetState *u, int l, const Vol &v, float *dx)
{
  const ConvSrc g = { u->G, kDesc[l].cout, 0 };
  const ConvSrc none = { nullptr, 0, 0 };
  if (tc_ok(u, v, kDesc[l].cin, kDesc[l].cout, 0))
    return tc_conv(u->G, kDesc[l].cout, nullptr, 0, v.B, v.Z, v.Y, v.X, u->wt[l], kDesc[l].cin,
        nullptr, 0, TC_F32, dx, u->err);
  switch (kDesc[l].cin) {
  case 16: return conv_mma<16, false>(g, none, v, u->wt[l], nullptr, 0, dx);
  case 32: return conv_mma<32, false>(g, none, v, u->wt[l], nullptr, 0, dx);
  case 48: return conv_mma<48, false>(g, none, v, u->wt[l], nullptr, 0, dx);
  case 96: return conv_mma<96, false>(g, none, v, u->wt[l], nullptr, 0, dx);
  }
  fail(NUSIF_ERR_STATE, "unet: no input-gradient kernel for %d channels", kDesc[l].cin);
  return false;
}

// weight and bias gradients of a layer from G (or, for the output layer, the
// FP32 gradient g32 itself) and its input
bool wgrad(UNetState *u, int l, const ConvSrc &s0, const ConvSrc &s1, const Vol &v,
    const float *g32 = nullptr)
{
  const int co = kDesc[l].cout, ci = kDesc[l].cin;
  return ensure_partial(u, wgrad_scratch(co, ci, v.B, v.Z, v.Y, v.X)) &&
         wgrad_conv({ s0.p, s0.c, s0.up }, { s1.p, s1.c, s1.up }, u->G, g32, co, ci, v.B, v.Z, v.Y,
             v.X, u->partial, u->grad + u->w_off[l], u->grad + u->b_off[l]);
}

// the grid of the row-indexed kernels: 8-channel groups of a row, rows, planes
dim3 row_grid(const Vol &v, int C)
{
  const int64_t planes = (int64_t)v.B * v.Z;
  return dim3((v.X * (C / 8) + 127) / 128, v.Y, (unsigned)(planes < 65535 ? planes : 65535));
}

// n values, a multiple of 8
bool mask(const float *dy, const bf16 *y, int64_t n, bf16 *g)
{
  k_relu_mask<<<blocks_for(n / 8), 256, 0, stream()>>>(dy, y, n / 8, g);
  return launched("k_relu_mask");
}

bool pool(const bf16 *f, const Vol &cv, int C, bf16 *o)
{
  k_pool<<<row_grid(cv, C), 128, 0, stream()>>>(f, cv, C, o);
  return launched("k_pool");
}

bool pool_back_mask(const float *gf, const float *gc, const Vol &fv, int C, const bf16 *y, bf16 *g)
{
  k_pool_back_mask<<<row_grid(fv, C), 128, 0, stream()>>>(gf, gc, fv, C, y, g);
  return launched("k_pool_back_mask");
}

// a layer's input gradient, masked by its input y (the layer before's output):
// u->G becomes that layer's masked output gradient
bool dgrad_mask(UNetState *u, int l, const Vol &v, const bf16 *y)
{
  const int n = kDesc[l].cin, c = kDesc[l].cout;
  if (tc_ok(u, v, n, c, 0) && tc_conv_marches(n, c)) {
    if (!tc_conv(u->G, c, nullptr, 0, v.B, v.Z, v.Y, v.X, u->wt[l], n, nullptr, 0, TC_MASKED, u->G2,
            u->err, 0, y))
      return false;
    std::swap(u->G, u->G2);
    return true;
  }
  return dgrad(u, l, v, u->F1) && mask(u->F1, y, n * v.cells(), u->G);
}

// the gradient of a concat [up(coarse) Cu, skip Cs]: the skip part to dskip,
// the upsampled part masked by the coarse layer's output y to u->G
bool dgrad_concat(UNetState *u, int l, const Vol &v, int Cu, int Cs, const bf16 *y, float *dskip)
{
  const int n = kDesc[l].cin, c = kDesc[l].cout;
  const Vol cv = { v.B, v.Z / 2, v.Y / 2, v.X / 2 };
  const bool split = Cu == 32 && Cs == 16 && tc_ok(u, v, n, c, 0) && tc_conv_marches(n, c);
  if (split) {
    if (!tc_conv(u->G, c, nullptr, 0, v.B, v.Z, v.Y, v.X, u->wt[l], n, nullptr, 0, TC_SPLIT, u->F1,
            u->err, 0, nullptr, dskip))
      return false;
  } else {
    const int64_t groups = v.cells() * (Cs / 8);
    if (!dgrad(u, l, v, u->F1)) return false;
    k_skip_part<<<blocks_for(groups), 256, 0, stream()>>>(u->F1, groups, Cu, Cs, dskip);
    if (!launched("k_skip_part")) return false;
  }
  k_up_back_mask<<<row_grid(cv, Cu), 128, 0, stream()>>>(u->F1, split ? Cu : n, cv, Cu, y, u->G);
  return launched("k_up_back_mask");
}

Vol half(const Vol &v) { return { v.B, v.Z / 2, v.Y / 2, v.X / 2 }; }

bool refresh_bf16(UNetState *u)
{
  for (int l = 0; l < kLayers; l++) {
    const int n = 27 * kDesc[l].cout * kDesc[l].cin;
    k_layer_bf16<<<(n + 255) / 256, 256, 0, stream()>>>(u->master + u->w_off[l], kDesc[l].cout,
        kDesc[l].cin, u->wb[l], u->wt[l]);
    if (!launched("k_layer_bf16")) return false;
  }
  k_pad_weights16<<<27, 256, 0, stream()>>>(u->master + u->w_off[L_E0A], 16, 2, u->w_first16);
  if (!launched("k_pad_weights16")) return false;
  k_pad_weights16<<<27, 256, 0, stream()>>>(u->master + u->w_off[L_OUT], 1, 16, u->w_last16);
  return launched("k_pad_weights16");
}

}  // namespace

// forward pass on the workspace input u->x (BF16) -> u->out (FP32)
bool unet_forward(UNetState *u)
{
  const Vol v0 = u->vol, v1 = half(v0), v2 = half(v1);
  const int64_t n0 = v0.cells();
  const ConvSrc none = { nullptr, 0, 0 };
  if (tc_ok(u, v0, 16, 16, 0)) {
    if (!tc_conv(u->x16, 16, nullptr, 0, v0.B, v0.Z, v0.Y, v0.X, u->w_first16, 16,
            u->master + u->b_off[L_E0A], 1, TC_BF16, u->e0a, u->err))
      return false;
  } else {
    k_conv_first<<<(unsigned)((n0 + 255) / 256), 256, 0, stream()>>>(u->x, v0, u->wb[L_E0A],
        u->master + u->b_off[L_E0A], u->e0a);
    if (!launched("k_conv_first")) return false;
  }
  if (!fwd(u, L_E0B, { u->e0a, 16, 0 }, none, v0, u->e0b)) return false;
  if (!pool(u->e0b, v1, 16, u->p0)) return false;
  if (!fwd(u, L_E1A, { u->p0, 16, 0 }, none, v1, u->e1a)) return false;
  if (!fwd(u, L_E1B, { u->e1a, 32, 0 }, none, v1, u->e1b)) return false;
  if (!pool(u->e1b, v2, 32, u->p1)) return false;
  if (!fwd(u, L_E2A, { u->p1, 32, 0 }, none, v2, u->e2a)) return false;
  if (!fwd(u, L_D1A, { u->e2a, 64, 1 }, { u->e1b, 32, 0 }, v1, u->d1a)) return false;
  if (!fwd(u, L_D1B, { u->d1a, 32, 0 }, none, v1, u->d1b)) return false;
  if (!fwd(u, L_D0A, { u->d1b, 32, 1 }, { u->e0b, 16, 0 }, v0, u->d0a)) return false;
  if (!fwd(u, L_D0B, { u->d0a, 16, 0 }, none, v0, u->d0b)) return false;
  if (tc_ok(u, v0, 16, 16, 0))
    return tc_conv(u->d0b, 16, nullptr, 0, v0.B, v0.Z, v0.Y, v0.X, u->w_last16, 16,
        u->master + u->b_off[L_OUT], 0, TC_ONE, u->out, u->err);
  k_conv_last<<<(unsigned)((n0 + 255) / 256), 256, 0, stream()>>>(u->d0b, v0, u->wb[L_OUT],
      u->master + u->b_off[L_OUT], u->out);
  return launched("k_conv_last");
}

// loss against `target` and the gradient of every parameter into u->grad
bool unet_backward(UNetState *u, const float *target)
{
  const Vol v0 = u->vol, v1 = half(v0), v2 = half(v1);
  const int64_t n0 = v0.cells();
  const ConvSrc none = { nullptr, 0, 0 };
  const int64_t lchunk = (n0 + 1023) / 1024 < 256 ? 256 : (n0 + 1023) / 1024;
  const int lblocks = (int)((n0 + lchunk - 1) / lchunk);
  k_mse<<<lblocks, 256, 0, stream()>>>(u->out, target, n0, lchunk, u->dout, u->loss_partial);
  if (!launched("k_mse")) return false;
  k_fold_loss<<<1, 256, 0, stream()>>>(u->loss_partial, lblocks, n0, u->loss);
  if (!launched("k_fold_loss")) return false;
  // out
  if (!wgrad(u, L_OUT, { u->d0b, 16, 0 }, none, v0, u->dout)) return false;
  k_conv_last_dgrad<<<(unsigned)((n0 / 4 + 127) / 128), 128, 0, stream()>>>(u->dout, v0,
      u->wb[L_OUT], u->d0b, u->G);
  if (!launched("k_conv_last_dgrad")) return false;
  // d0b
  if (!wgrad(u, L_D0B, { u->d0a, 16, 0 }, none, v0) || !dgrad_mask(u, L_D0B, v0, u->d0a)) return false;
  // d0a (input concat [up(d1b) 32, e0b 16])
  if (!wgrad(u, L_D0A, { u->d1b, 32, 1 }, { u->e0b, 16, 0 }, v0) ||
      !dgrad_concat(u, L_D0A, v0, 32, 16, u->d1b, u->Fe0b))
    return false;
  // d1b
  if (!wgrad(u, L_D1B, { u->d1a, 32, 0 }, none, v1) || !dgrad_mask(u, L_D1B, v1, u->d1a)) return false;
  // d1a (input concat [up(e2a) 64, e1b 32])
  if (!wgrad(u, L_D1A, { u->e2a, 64, 1 }, { u->e1b, 32, 0 }, v1) ||
      !dgrad_concat(u, L_D1A, v1, 64, 32, u->e2a, u->Fe1b))
    return false;
  // e2a, whose input is the pooled e1b
  if (!wgrad(u, L_E2A, { u->p1, 32, 0 }, none, v2) || !dgrad(u, L_E2A, v2, u->F2) ||
      !pool_back_mask(u->Fe1b, u->F2, v1, 32, u->e1b, u->G))
    return false;
  // e1b
  if (!wgrad(u, L_E1B, { u->e1a, 32, 0 }, none, v1) || !dgrad_mask(u, L_E1B, v1, u->e1a)) return false;
  // e1a, whose input is the pooled e0b
  if (!wgrad(u, L_E1A, { u->p0, 16, 0 }, none, v1) || !dgrad(u, L_E1A, v1, u->F2) ||
      !pool_back_mask(u->Fe0b, u->F2, v0, 16, u->e0b, u->G))
    return false;
  // e0b
  if (!wgrad(u, L_E0B, { u->e0a, 16, 0 }, none, v0) || !dgrad_mask(u, L_E0B, v0, u->e0a)) return false;
  // e0a (no input gradient)
  return wgrad(u, L_E0A, { u->x16, 16, 0 }, none, v0);
}

bool unet_set_input(UNetState *u, const float *x, const Vol &v)
{
  if (!ensure_workspace(u, v)) return false;
  k_input_bf16<<<blocks_for(v.cells()), 256, 0, stream()>>>(x, v.cells(), u->x, u->x16);
  return launched("k_input_bf16");
}

}  // namespace nusif

using namespace nusif;

struct NusifUNet {
  UNetState s;
};

namespace {

// splitmix64 + Box-Muller: He-normal initial weights, zero biases
struct Rng {
  uint64_t s;
  uint64_t next()
  {
    uint64_t z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
  }
  double uniform() { return ((next() >> 11) + 0.5) * (1.0 / 9007199254740992.0); }
  double normal()
  {
    const double a = uniform(), b = uniform();
    return sqrt(-2.0 * log(a)) * cos(6.283185307179586 * b);
  }
};

NusifUNet *checked(NusifUNet *n)
{
  if (!n) fail(NUSIF_ERR_ARG, "unet: null network");
  return n;
}

// the tensor-core kernels' error flag (a bounded wait that ran out); synchronises
bool tc_clean(UNetState *u)
{
  int e = 0;
  if (!cuda_ok(cudaMemcpyAsync(&e, u->err, sizeof(int), cudaMemcpyDeviceToHost, stream()),
          "unet error flag") ||
      !cuda_ok(cudaStreamSynchronize(stream()), "unet error flag"))
    return false;
  if (e) {
    cudaMemsetAsync(u->err, 0, sizeof(int), stream());
    fail(NUSIF_ERR_CUDA, "unet: a tensor-core convolution timed out waiting for its operands");
    return false;
  }
  return true;
}

}  // namespace

namespace nusif {

bool unet_infer(NusifUNet *net, const float *x, int Z, int Y, int X, const float **out)
{
  UNetState *u = &net->s;
  const Vol v = { 1, Z, Y, X };
  if (!unet_set_input(u, x, v) || !unet_forward(u)) return false;
  *out = u->out;
  return true;
}

}  // namespace nusif

extern "C" {

NusifUNet *nusifUNetCreate(unsigned long long seed)
{
  NusifUNet *n = new NusifUNet();
  UNetState *u = &n->s;
  int64_t o = 0;
  for (int l = 0; l < kLayers; l++) {
    u->w_off[l] = o;
    o += 27 * kDesc[l].cout * kDesc[l].cin;
    u->b_off[l] = o;
    o += kDesc[l].cout;
  }
  u->nparam = o;
  std::vector<float> h(o, 0.0f);
  Rng rng{ seed };
  for (int l = 0; l < kLayers; l++) {
    const double sd = sqrt(2.0 / (27.0 * kDesc[l].cin));
    for (int64_t i = 0; i < 27 * kDesc[l].cout * kDesc[l].cin; i++)
      h[u->w_off[l] + i] = (float)(sd * rng.normal());
  }
  bool ok = cuda_ok(cudaMalloc(&u->master, o * sizeof(float)), "cudaMalloc(unet)") &&
            cuda_ok(cudaMalloc(&u->grad, o * sizeof(float)), "cudaMalloc(unet)") &&
            cuda_ok(cudaMalloc(&u->m, o * sizeof(float)), "cudaMalloc(unet)") &&
            cuda_ok(cudaMalloc(&u->v, o * sizeof(float)), "cudaMalloc(unet)") &&
            cuda_ok(cudaMalloc(&u->loss, sizeof(float)), "cudaMalloc(unet)") &&
            cuda_ok(cudaMalloc(&u->err, sizeof(int)), "cudaMalloc(unet)") &&
            cuda_ok(cudaMemset(u->err, 0, sizeof(int)), "unet init");
  ok = ok && cuda_ok(cudaMalloc(&u->w_first16, 27 * 256 * sizeof(bf16)), "cudaMalloc(unet)") &&
       cuda_ok(cudaMalloc(&u->w_last16, 27 * 256 * sizeof(bf16)), "cudaMalloc(unet)");
  for (int l = 0; ok && l < kLayers; l++) {
    const size_t nw = 27 * kDesc[l].cout * kDesc[l].cin;
    ok = cuda_ok(cudaMalloc(&u->wb[l], nw * sizeof(bf16)), "cudaMalloc(unet)") &&
         cuda_ok(cudaMalloc(&u->wt[l], nw * sizeof(bf16)), "cudaMalloc(unet)");
  }
  ok = ok && cuda_ok(cudaMemcpy(u->master, h.data(), o * sizeof(float), cudaMemcpyHostToDevice),
                 "unet init") &&
       cuda_ok(cudaMemset(u->grad, 0, o * sizeof(float)), "unet init") &&
       cuda_ok(cudaMemset(u->m, 0, o * sizeof(float)), "unet init") &&
       cuda_ok(cudaMemset(u->v, 0, o * sizeof(float)), "unet init") && refresh_bf16(u) &&
       cuda_ok(cudaStreamSynchronize(stream()), "unet init");
  if (!ok) {
    nusifUNetFree(n);
    return nullptr;
  }
  return n;
}

void nusifUNetFree(NusifUNet *n)
{
  if (!n) return;
  UNetState *u = &n->s;
  cudaDeviceSynchronize();
  free_workspace(u);
  if (u->partial) cudaFree(u->partial);
  for (float *p : { u->master, u->grad, u->m, u->v, u->loss })
    if (p) cudaFree(p);
  if (u->err) cudaFree(u->err);
  if (u->w_first16) cudaFree(u->w_first16);
  if (u->w_last16) cudaFree(u->w_last16);
  for (int l = 0; l < kLayers; l++) {
    if (u->wb[l]) cudaFree(u->wb[l]);
    if (u->wt[l]) cudaFree(u->wt[l]);
  }
  delete n;
}

long long nusifUNetParamCount(const NusifUNet *n) { return n ? n->s.nparam : 0; }

int nusifUNetGetParams(const NusifUNet *n, float *host, long long count)
{
  if (!checked(const_cast<NusifUNet *>(n)) || !host || count != n->s.nparam) {
    fail(NUSIF_ERR_ARG, "nusifUNetGetParams: need %lld values", n ? (long long)n->s.nparam : 0LL);
    return NUSIF_ERR_ARG;
  }
  if (!cuda_ok(cudaMemcpyAsync(host, n->s.master, count * sizeof(float), cudaMemcpyDeviceToHost,
                   stream()),
          "unet params") ||
      !cuda_ok(cudaStreamSynchronize(stream()), "unet params"))
    return NUSIF_ERR_CUDA;
  return NUSIF_OK;
}

int nusifUNetGetGrads(const NusifUNet *n, float *host, long long count)
{
  if (!checked(const_cast<NusifUNet *>(n)) || !host || count != n->s.nparam) {
    fail(NUSIF_ERR_ARG, "nusifUNetGetGrads: need %lld values", n ? (long long)n->s.nparam : 0LL);
    return NUSIF_ERR_ARG;
  }
  if (!cuda_ok(cudaMemcpyAsync(host, n->s.grad, count * sizeof(float), cudaMemcpyDeviceToHost,
                   stream()),
          "unet grads") ||
      !cuda_ok(cudaStreamSynchronize(stream()), "unet grads"))
    return NUSIF_ERR_CUDA;
  return NUSIF_OK;
}

int nusifUNetSetParams(NusifUNet *n, const float *host, long long count)
{
  if (!checked(n) || !host || count != n->s.nparam) {
    fail(NUSIF_ERR_ARG, "nusifUNetSetParams: need %lld values", n ? (long long)n->s.nparam : 0LL);
    return NUSIF_ERR_ARG;
  }
  UNetState *u = &n->s;
  if (!cuda_ok(cudaMemcpyAsync(u->master, host, count * sizeof(float), cudaMemcpyHostToDevice,
                   stream()),
          "unet params") ||
      !cuda_ok(cudaMemsetAsync(u->m, 0, count * sizeof(float), stream()), "unet adam") ||
      !cuda_ok(cudaMemsetAsync(u->v, 0, count * sizeof(float), stream()), "unet adam") ||
      !refresh_bf16(u) || !cuda_ok(cudaStreamSynchronize(stream()), "unet params"))
    return NUSIF_ERR_CUDA;
  u->adam_t = 0;
  return NUSIF_OK;
}

int nusifUNetForward(NusifUNet *n, const float *x, int B, int Z, int Y, int X, float *out)
{
  if (!checked(n) || !x || !out) return NUSIF_ERR_ARG;
  UNetState *u = &n->s;
  const Vol v = { B, Z, Y, X };
  if (!unet_set_input(u, x, v) || !unet_forward(u)) return has_error() ? NUSIF_ERR_CUDA : NUSIF_ERR_ARG;
  if (!cuda_ok(cudaMemcpyAsync(out, u->out, v.cells() * sizeof(float), cudaMemcpyDeviceToDevice,
                   stream()),
          "unet output"))
    return NUSIF_ERR_CUDA;
  return tc_clean(u) ? NUSIF_OK : NUSIF_ERR_CUDA;
}

int nusifUNetSetTensorCore(NusifUNet *n, int mode)
{
  if (!checked(n) || (mode != 0 && mode != 1)) {
    fail(NUSIF_ERR_ARG, "nusifUNetSetTensorCore: mode 0 (mma.sync) or 1 (tcgen05)");
    return NUSIF_ERR_ARG;
  }
  n->s.use_tc = mode;
  return NUSIF_OK;
}

int nusifUNetTrainStep(NusifUNet *n, const float *x, const float *target, int B, int Z, int Y,
    int X, float lr, int update, float *loss_host)
{
  if (!checked(n) || !x || !target) return NUSIF_ERR_ARG;
  UNetState *u = &n->s;
  const Vol v = { B, Z, Y, X };
  if (!unet_set_input(u, x, v) || !unet_forward(u) || !unet_backward(u, target))
    return NUSIF_ERR_CUDA;
  if (update) {
    u->adam_t++;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.0f - powf(b1, (float)u->adam_t), c2 = 1.0f - powf(b2, (float)u->adam_t);
    k_adam<<<blocks_for(u->nparam), 256, 0, stream()>>>(u->master, u->grad, u->m, u->v, u->nparam,
        lr, b1, b2, 1e-8f, c1, c2);
    if (!launched("k_adam") || !refresh_bf16(u)) return NUSIF_ERR_CUDA;
  }
  if (loss_host) {
    if (!cuda_ok(cudaMemcpyAsync(loss_host, u->loss, sizeof(float), cudaMemcpyDeviceToHost, stream()),
            "unet loss") ||
        !cuda_ok(cudaStreamSynchronize(stream()), "unet loss"))
      return NUSIF_ERR_CUDA;
    if (!tc_clean(u)) return NUSIF_ERR_CUDA;
  }
  return NUSIF_OK;
}

}  // extern "C"
