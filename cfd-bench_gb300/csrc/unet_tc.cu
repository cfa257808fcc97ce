// 3x3x3 convolutions of the U-Net on the 5th-generation tensor cores
// (tcgen05.mma, accumulators in tensor memory, operands staged by TMA).
//
// Implicit GEMM: M = 128 cells of one z-plane (a tile of 16 x-columns by 8
// y-rows), N = output channels, K = 27 taps x input channels. The tile's rows
// are ordered x-major over 8-cell y-columns, so each x-column is one 8-row
// swizzle atom of the K-major operand layout. A stage carries one (dz, dy)
// row of taps: per source one TMA tiled load of the 18 x-columns x 8 y-rows
// around the tile (x from x0 - 1 to x0 + 16, through a tensor map whose
// second dimension is y and third x, so the box lands column by column), and
// one load of the row's three tap weights [3][N][C]. The three dx taps of the
// row read that one box through descriptors offset by 0, 1 and 2 atoms, so a
// cell row is loaded once per (dz, dy) instead of once per tap. Out-of-range
// x and y read as zero, which is the convolution's zero padding; a dz plane
// outside the volume is skipped for the whole tile. The swizzle is the one
// whose span is the cell row (32, 64 or 128 bytes for 16, 32 or 64 channels),
// which is also the canonical K-major operand layout for that span (8-row
// atoms; stride offset 8 rows). The MMA thread issues one tcgen05.mma
// (kind::f16, BF16 x BF16 -> FP32, M = 128, N = channels out, K = 16) per 16
// input channels per tap, the descriptors advanced by 32 bytes along the
// swizzled row, and commits the stage back to the producer. Accumulators are
// double-buffered in tensor memory, so four epilogue warps drain one tile
// (tcgen05.ld, bias, ReLU, BF16 or FP32 rows) while the next tile's products
// accumulate.
//
// Two sources (the decoder's concat) are two K ranges of the same tile.
// Every mbarrier wait is bounded (about one second); a wait that runs out
// sets an error flag the host reads, the warps stop issuing work, wait
// (bounded) for the copies and products already issued, free tensor memory
// and return.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>

#include <cstdint>
#include <cstdlib>
#include <cstdio>

#include "nusif_internal.h"
#include "unet_tc.h"

namespace nusif {
namespace {

constexpr int kTileM = 128;
constexpr int kTileX = 16, kTileY = 8;  // tile: 16 x-columns of 8 y-cells
constexpr int kBoxX = kTileX + 2;       // loaded columns: the tile and one on each side
constexpr int kThreads = 192;  // warp 0 TMA producer, warp 1 MMA issuer, warps 2-5 epilogue
constexpr int kMaxStages = 16;
constexpr uint32_t kBarBytes = 512;  // barrier and flag region at the start of shared memory
constexpr long long kWaitClocks = 2000000000ll;  // bound of every mbarrier wait: about a second

struct TcParams {
  int N;                 // output channels (MMA N)
  int C0, C1;            // channels of source 0 and source 1 (0: none): 16, 32 or 64
  uint32_t a_off[2], b_off[2];  // offsets of each source's cell box and tap weights in a stage
  uint32_t atom[2];      // bytes of one x-column (8 cell rows) of each source
  uint32_t wtap[2];      // bytes of one tap's weights [N][C] of each source
  uint32_t stage_bytes, tx_bytes;
  int X, Y, Z, B;        // volume
  int tx, ty;            // tiles per row (X / 16) and per column (Y / 8)
  int ntiles;
  int stages;
  int tmem_cols;         // allocated tensor-memory columns (>= 2 N, power of two)
  uint32_t idesc;        // instruction descriptor
  const float *bias;     // [N] or nullptr
  int relu;
  int out_bf16;
  void *out;             // [cells][N]
  int *err;
};

__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity)
{
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// the same test, the thread suspended (no issue slots) until the phase
// completes or about `hint_ns` pass
__device__ __forceinline__ bool mbar_try_sleep(uint32_t bar, uint32_t parity, uint32_t hint_ns)
{
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(hint_ns)
      : "memory");
  return ok != 0;
}

// wait for the phase of `parity` to complete; false after the time bound or
// when another warp has raised the abort flag. Waiting threads sleep in the
// barrier rather than spin, so the single-thread producer and MMA issuer of
// the block's other warps keep their issue slots; the abort flag and the
// clock are read every 8th round.
__device__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag, int *err)
{
  if (mbar_try(bar, parity)) return true;
  long long t0 = 0;
  for (uint32_t round = 1;; round++) {
    if (mbar_try_sleep(bar, parity, 20000u)) return true;
    if ((round & 7u) == 0) {
      if (*abort_flag) return false;
      if (t0 == 0) t0 = clock64();
      if (clock64() - t0 > kWaitClocks) {
        *abort_flag = 1;
        atomicExch(err, 1);
        return false;
      }
    }
  }
}

// bounded wait used while draining after an abort (does not re-raise it)
__device__ void mbar_drain(uint32_t bar, uint32_t parity)
{
  const long long t0 = clock64();
  while (!mbar_try(bar, parity) && clock64() - t0 < kWaitClocks) {
  }
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count)
{
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes)
{
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap *map, uint32_t bar,
    int c0, int c1, int c2, int c3)
{
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar)
      : "memory");
}

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *map, uint32_t bar,
    int c0, int c1, int c2)
{
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
      : "memory");
}

// shared-memory matrix descriptor, K-major, rows of `row_bytes` (32, 64 or
// 128) in the swizzle of that span: stride offset = one 8-row atom, leading
// offset unused (1), base offset 0 (atoms 1024-byte aligned)
__device__ __forceinline__ uint64_t smem_desc_sw(uint32_t addr, uint32_t row_bytes)
{
  const uint64_t mode = row_bytes == 128u ? 2u : row_bytes == 64u ? 4u : 6u;
  uint64_t d = (uint64_t)((addr & 0x3FFFFu) >> 4);
  d |= 1ull << 16;                                      // leading byte offset (unused)
  d |= (uint64_t)(((8u * row_bytes) >> 4) & 0x3FFFu) << 32;  // stride byte offset
  d |= 1ull << 46;  // descriptor version of this architecture
  d |= mode << 61;  // swizzle mode
  return d;
}

__device__ __forceinline__ void mma_f16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc,
    uint32_t accumulate)
{
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void mma_commit(uint32_t bar)
{
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
      : "memory");
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 16 consecutive FP32 columns of this warp's 32 lanes (one row per thread)
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16])
{
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
        "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
#pragma unroll
  for (int q = 0; q < 16; q++) v[q] = __uint_as_float(r[q]);
}

__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ uint32_t pack2(float a, float b)
{
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t *>(&v);
}

struct Tile {
  int x0, y0, zb, z;
};

__device__ __forceinline__ Tile tile_of(const TcParams &P, int t)
{
  Tile r;
  r.x0 = (t % P.tx) * kTileX;
  const int rest = t / P.tx;
  r.y0 = (rest % P.ty) * kTileY;
  r.zb = rest / P.ty;
  r.z = r.zb % P.Z;
  return r;
}

template <int NCH>  // output channels, a multiple of 16
__global__ void __launch_bounds__(kThreads) k_conv_tc(const __grid_constant__ CUtensorMap tm_a0,
    const __grid_constant__ CUtensorMap tm_a1, const __grid_constant__ CUtensorMap tm_w0,
    const __grid_constant__ CUtensorMap tm_w1, const TcParams P)
{
  extern __shared__ __align__(1024) unsigned char smem[];
  // [0, kBarBytes): barriers, then the tensor-memory address and the abort
  // flag; stages from the first 1024-byte boundary after that
  static_assert((2 * kMaxStages + 4) * 8 + 8 <= kBarBytes, "barriers overlap the flags");
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem);
  uint64_t *full = bars, *empty = bars + kMaxStages, *acc_full = bars + 2 * kMaxStages,
           *acc_empty = bars + 2 * kMaxStages + 2;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + kBarBytes - 8);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + kBarBytes - 4);
  // stages start at the first 1024-byte boundary past the barriers (TMA destinations
  // need 128-byte alignment)
  const uint32_t sbase = smem_u32(smem);
  unsigned char *stage_base = smem + (((sbase + kBarBytes + 1023u) & ~1023u) - sbase);
  const uint32_t stage_bytes = P.stage_bytes;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < P.stages; s++) {
      mbar_init(smem_u32(full + s), 1);
      mbar_init(smem_u32(empty + s), 1);
    }
    for (int b = 0; b < 2; b++) {
      mbar_init(smem_u32(acc_full + b), 1);
      mbar_init(smem_u32(acc_empty + b), 128);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {  // tensor memory for two accumulators
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(P.tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0 && lane == 0) {
    // ---------------- TMA producer ----------------
    bool armed[kMaxStages];
    uint32_t armed_par[kMaxStages];
    for (int s = 0; s < kMaxStages; s++) armed[s] = false;
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int t = blockIdx.x; ok && t < P.ntiles; t += gridDim.x) {
      const Tile tl = tile_of(P, t);
      for (int row = 0; row < 9; row++) {  // (dz, dy) rows of taps; a stage per row
        const int dz = row / 3 - 1, dy = row % 3 - 1;
        if (tl.z + dz < 0 || tl.z + dz >= P.Z) continue;
        if (!mbar_wait(smem_u32(empty + stage), phase ^ 1u, abort_flag, P.err)) {
          ok = false;
          break;
        }
        armed[stage] = false;
        const uint32_t fb = smem_u32(full + stage);
        const uint32_t sa = smem_u32(stage_base + (size_t)stage * stage_bytes);
        mbar_expect_tx(fb, P.tx_bytes);
        // the box (C, 8 y, 18 x) at y0 + dy, x0 - 1; the row's three taps' weights
        tma_load_4d(sa + P.a_off[0], &tm_a0, fb, 0, tl.y0 + dy, tl.x0 - 1, tl.zb + dz);
        tma_load_3d(sa + P.b_off[0], &tm_w0, fb, 0, 0, 3 * row);
        if (P.C1 > 0) {
          tma_load_4d(sa + P.a_off[1], &tm_a1, fb, 0, tl.y0 + dy, tl.x0 - 1, tl.zb + dz);
          tma_load_3d(sa + P.b_off[1], &tm_w1, fb, P.C0, 0, 3 * row);
        }
        armed[stage] = true;
        armed_par[stage] = phase;
        if (++stage == P.stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    if (!ok)  // let the copies already issued land before the shared memory goes away
      for (int s = 0; s < P.stages; s++)
        if (armed[s]) mbar_drain(smem_u32(full + s), armed_par[s]);
  } else if (warp == 1 && lane == 0) {
    // ---------------- MMA issuer ----------------
    int stage = 0;
    uint32_t phase = 0;
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    bool issued = false;
    for (int t = blockIdx.x; ok && t < P.ntiles; t += gridDim.x) {
      const Tile tl = tile_of(P, t);
      if (!mbar_wait(smem_u32(acc_empty + acc), acc_phase ^ 1u, abort_flag, P.err)) {
        ok = false;
        break;
      }
      fence_after();
      const uint32_t d = tmem + (uint32_t)(acc * (P.tmem_cols / 2));
      uint32_t accumulate = 0;
      for (int row = 0; row < 9; row++) {
        const int dz = row / 3 - 1;
        if (tl.z + dz < 0 || tl.z + dz >= P.Z) continue;
        if (!mbar_wait(smem_u32(full + stage), phase, abort_flag, P.err)) {
          ok = false;
          break;
        }
        fence_after();
        const uint32_t sa = smem_u32(stage_base + (size_t)stage * stage_bytes);
        // the descriptors' start-address field is (address >> 4) in 14 bits;
        // every operand lies below 256 KB, so offsets add to it without carry
        uint64_t a0[2], b0[2];
        uint32_t da[2], db[2];
        int ks[2];
        for (int src = 0; src < 2; src++) {
          ks[src] = (src == 0 ? P.C0 : P.C1) / 16;
          const uint32_t rb = 32u * (uint32_t)ks[src];
          a0[src] = smem_desc_sw(sa + P.a_off[src], rb);
          b0[src] = smem_desc_sw(sa + P.b_off[src], rb);
          da[src] = P.atom[src] >> 4;
          db[src] = P.wtap[src] >> 4;
        }
        for (int q = 0; q < 3; q++) {  // dx = q - 1: the box read q atoms in
          for (int src = 0; src < 2; src++) {
            for (int j = 0; j < ks[src]; j++) {
              mma_f16(d, a0[src] + (uint64_t)(q * da[src] + 2u * j),
                  b0[src] + (uint64_t)(q * db[src] + 2u * j), P.idesc, accumulate);
              accumulate = 1;
              issued = true;
            }
          }
        }
        mma_commit(smem_u32(empty + stage));
        if (++stage == P.stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
      if (!ok) break;
      mma_commit(smem_u32(acc_full + acc));
      if (++acc == 2) {
        acc = 0;
        acc_phase ^= 1u;
      }
    }
    if (!ok && issued) {  // wait for every product already issued
      mma_commit(smem_u32(acc_full + acc));
      mbar_drain(smem_u32(acc_full + acc), acc_phase);
    }
  } else if (warp >= 2) {
    // ---------------- epilogue: tensor memory -> bias, ReLU -> global ----------------
    const int q = warp & 3;  // this warp may read lanes 32q .. 32q + 31
    const int row = 32 * q + lane;
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int t = blockIdx.x; t < P.ntiles; t += gridDim.x) {
      // warp-uniform: the tensor-memory loads below need the whole warp
      const bool ready = mbar_wait(smem_u32(acc_full + acc), acc_phase, abort_flag, P.err);
      if (!__all_sync(0xffffffffu, ready)) break;
      fence_after();
      float v[NCH];
#pragma unroll
      for (int c = 0; c < NCH; c += 16) {
        float part[16];
        tmem_ld16(tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(acc * (P.tmem_cols / 2) + c),
            part);
#pragma unroll
        for (int e = 0; e < 16; e++) v[c + e] = part[e];
      }
      tmem_wait_ld();
      fence_before();
      mbar_arrive(smem_u32(acc_empty + acc));
      // accumulator row = x-column * 8 + y within the tile
      const Tile tl = tile_of(P, t);
      const int64_t cell =
          ((int64_t)tl.zb * P.Y + tl.y0 + (row & 7)) * P.X + tl.x0 + (row >> 3);
#pragma unroll
      for (int c = 0; c < NCH; c++) {
        const float x = v[c] + (P.bias ? __ldg(P.bias + c) : 0.0f);
        v[c] = P.relu ? fmaxf(x, 0.0f) : x;
      }
      if (P.out_bf16) {
        uint4 *o = reinterpret_cast<uint4 *>(static_cast<__nv_bfloat16 *>(P.out) + cell * NCH);
#pragma unroll
        for (int c = 0; c < NCH; c += 8)
          o[c / 8] = make_uint4(pack2(v[c], v[c + 1]), pack2(v[c + 2], v[c + 3]),
              pack2(v[c + 4], v[c + 5]), pack2(v[c + 6], v[c + 7]));
      } else {
        float4 *o = reinterpret_cast<float4 *>(static_cast<float *>(P.out) + cell * NCH);
#pragma unroll
        for (int c = 0; c < NCH; c += 4) o[c / 4] = make_float4(v[c], v[c + 1], v[c + 2], v[c + 3]);
      }
      if (++acc == 2) {
        acc = 0;
        acc_phase ^= 1u;
      }
    }
  }
  fence_before();
  __syncthreads();
  if (warp == 0) {
    __syncwarp();
    fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(P.tmem_cols)
                 : "memory");
  }
}

// ------------------------------------------------------------------ marching form
//
// The layers of up to 48 channels on either side (every full-resolution layer,
// forward and input gradient). k_conv_tc loads a tile's neighbourhood nine
// times, in boxes of 32- to 128-byte rows, and that many short rows, not the
// products, set its pace (about 5000 cycles a tile of a 16 -> 16 layer). Here
// a block owns a column of 8 x 16 cells and marches over the planes. A plane
// (10 x 18 cells around the column) is fetched once, by 16-byte cp.async, and
// used once: its products go to the three output planes it belongs to, as one
// tcgen05.mma per (dy, dx) and 16 channels with N = 3 x channels out, the
// weights of the three dz side by side. That also reads A from shared memory a
// third as often, which is what bounds a product of so few columns (128 rows of
// 32 bytes each time).
//
// The operand needs no copy per tap: a cell's 8-channel group is 16 bytes, eight
// cells along x are one 8 x 16-byte core matrix of the unswizzled K-major
// layout, the next eight rows of the operand are the next y, and a tap is an
// offset of the start address by whole cells. All weights stay in shared memory.
//
// Accumulators of the output planes are groups of N columns in a ring in tensor
// memory, so the window of three slides by N columns a plane (two products where
// it wraps). A group starts from zeros, which the epilogue stores after it has
// drained it. Every output is summed in the order of k_conv_tc (dz, dy, dx, then
// channels), so the results are the same bits.
constexpr int kColX = 8, kColY = 16;                // cells of a column
constexpr int kInX = kColX + 2, kInY = kColY + 2;   // and of the plane it reads
constexpr int kRowB = kInX * 16;                    // bytes of a y-row of one 8-channel group
constexpr int kGroupB = kInY * kRowB;               // bytes of one 8-channel group of a plane
constexpr int kSlotsC = 4;                          // planes in shared memory
constexpr int kMaxGroups = 8;
constexpr int kColThreads = 256;  // warp 0 products, 1-3 loads, 4-7 epilogue
constexpr int kLoaders = 96;

struct ColParams {
  const __nv_bfloat16 *s0, *s1;  // sources of C0 and C1 channels
  const __nv_bfloat16 *w;        // [27][N][C0 + C1]
  int C0, C1, up0;               // up0: source 0 at half resolution, read by nearest upsampling
  int X, Y, Z, B;
  int tx, ty;      // columns per row and per plane
  int zl, zt;      // planes of a march, marches per column
  int items;
  const float *bias;
  int relu, kind;  // TcOut
  void *out, *out2;
  const __nv_bfloat16 *mask;
  int *err;
};

struct March {
  int x0, y0, b, z0, z1;
};

__device__ __forceinline__ March march_of(const ColParams &P, int t)
{
  March m;
  m.x0 = (t % P.tx) * kColX;
  int r = t / P.tx;
  m.y0 = (r % P.ty) * kColY;
  r /= P.ty;
  m.z0 = (r % P.zt) * P.zl;
  m.z1 = min(m.z0 + P.zl, P.Z) - 1;
  m.b = r / P.zt;
  return m;
}

// unswizzled K-major descriptor: lead = bytes between the two 8-element halves
// of K, stride = bytes between groups of 8 rows
__device__ __forceinline__ uint64_t smem_desc_plain(uint32_t addr, uint32_t lead, uint32_t stride)
{
  uint64_t d = (uint64_t)((addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)((lead >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((stride >> 4) & 0x3FFFu) << 32;
  d |= 1ull << 46;
  return d;
}

__device__ __forceinline__ void tmem_zero16(uint32_t taddr)
{
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1};" ::"r"(taddr),
      "r"(0u)
      : "memory");
}

__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void fence_proxy() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// NCH output and CIN input channels, 16, 32 or 48 each
template <int NCH, int CIN>
struct Col {
  static constexpr int kHalves = CIN / 8;                   // 8-channel groups
  static constexpr uint32_t kSlotB = kHalves * kGroupB;
  static constexpr uint32_t kTapB = kHalves * 3 * NCH * 16;  // weights of one (dy, dx)
  static constexpr uint32_t kWeightB = 9 * kTapB;
  static constexpr int kCols = NCH == 16 ? 128 : 256;  // tensor-memory columns of a block
  static constexpr int kGroups = kCols / NCH < kMaxGroups ? kCols / NCH : kMaxGroups;
  static constexpr size_t kSmem = kBarBytes + 128 + kWeightB + kSlotsC * kSlotB;
};

template <int NCH, int CIN>
__global__ void __launch_bounds__(kColThreads) k_conv_col(const ColParams P)
{
  using L = Col<NCH, CIN>;
  extern __shared__ __align__(1024) unsigned char smem[];
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem);
  uint64_t *full = bars, *empty = bars + kSlotsC, *acc_full = bars + 2 * kSlotsC,
           *acc_empty = acc_full + kMaxGroups;
  static_assert((2 * kSlotsC + 2 * kMaxGroups) * 8 + 8 <= kBarBytes, "barriers overlap the flags");
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + kBarBytes - 8);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + kBarBytes - 4);
  const uint32_t weights = smem_u32(smem) + kBarBytes, planes = weights + L::kWeightB;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    for (int s = 0; s < kSlotsC; s++) {
      mbar_init(smem_u32(full + s), kLoaders);
      mbar_init(smem_u32(empty + s), 1);
    }
    for (int g = 0; g < kMaxGroups; g++) {
      mbar_init(smem_u32(acc_full + g), 1);
      mbar_init(smem_u32(acc_empty + g), 128);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(L::kCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  // weights: per (dy, dx) and 8 channels, rows dz = +1, 0, -1 of N channels: the
  // row blocks of output planes p - 1, p, p + 1 for an input plane p
  for (int i = tid; i < 27 * NCH * L::kHalves; i += kColThreads) {
    const int h = i % L::kHalves, r = i / L::kHalves, n = r % NCH, tap = r / NCH;
    const int dz = tap / 9 - 1, dydx = tap % 9;
    const uint4 v = *reinterpret_cast<const uint4 *>(P.w + ((size_t)tap * NCH + n) * CIN + 8 * h);
    const uint32_t at = (uint32_t)(dydx * (int)L::kTapB + (h * 3 * NCH + (1 - dz) * NCH + n) * 16);
    *reinterpret_cast<uint4 *>(smem + kBarBytes + at) = v;
  }
  fence_proxy();
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = *tmem_slot;
  if (warp >= 4) {  // every group starts from zeros
    for (int c = 0; c < L::kGroups * NCH; c += 16)
      tmem_zero16(tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)c);
    tmem_wait_st();
  }
  fence_before();
  __syncthreads();
  fence_after();

  if (warp >= 1 && warp <= 3) {
    // ---------------- loads: one plane a slot ----------------
    // this thread's chunks (a cell's 8 channels) of a plane: where they go, and
    // per march where they come from (offset in the plane, -1: outside)
    constexpr int kPer = (kInY * kInX * L::kHalves + kLoaders - 1) / kLoaders;
    const int t0 = tid - 32;
    int slot = 0, prev = -1;
    uint32_t phase = 0;
    bool ok = true;
    for (int t = blockIdx.x; ok && t < P.items; t += gridDim.x) {
      const March m = march_of(P, t);
      const int p1 = min(m.z1 + 1, P.Z - 1);
      int from[kPer];
#pragma unroll
      for (int q = 0; q < kPer; q++) {
        const int i = t0 + q * kLoaders;
        const int h = i % L::kHalves, c = i / L::kHalves, cx = c % kInX, cy = c / kInX;
        const int x = m.x0 - 1 + cx, y = m.y0 - 1 + cy;
        const bool in = x >= 0 && x < P.X && y >= 0 && y < P.Y;
        const bool second = 8 * h >= P.C0;
        const int up = second ? 0 : P.up0;
        const int cell = (y >> up) * (P.X >> up) + (x >> up);
        from[q] = !in ? -1 : second ? cell * P.C1 + 8 * h - P.C0 : cell * P.C0 + 8 * h;
      }
      for (int p = max(m.z0 - 1, 0); p <= p1; p++) {
        if (!mbar_wait(smem_u32(empty + slot), phase ^ 1u, abort_flag, P.err)) {
          ok = false;
          break;
        }
        const int64_t zb = (int64_t)m.b * P.Z + p;
        const __nv_bfloat16 *const b0 =
            P.s0 + (P.up0 ? ((int64_t)m.b * (P.Z >> 1) + (p >> 1)) * (P.Y >> 1) * (P.X >> 1)
                          : zb * P.Y * P.X) * P.C0;
        const __nv_bfloat16 *const b1 = P.s1 + zb * P.Y * P.X * P.C1;
        const uint32_t dst0 = planes + (uint32_t)slot * L::kSlotB;
#pragma unroll
        for (int q = 0; q < kPer; q++) {
          const int i = t0 + q * kLoaders;
          const int h = i % L::kHalves, c = i / L::kHalves, cx = c % kInX, cy = c / kInX;
          if (q + 1 == kPer && i >= kInY * kInX * L::kHalves) continue;
          const bool in = from[q] >= 0;
          const __nv_bfloat16 *src = (8 * h >= P.C0 ? b1 : b0) + (in ? from[q] : 0);
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                           dst0 + (uint32_t)(h * kGroupB + cy * kRowB + cx * 16)),
                       "l"(src), "r"(in ? 16 : 0)
                       : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (prev >= 0) {  // the plane before this one is in
          asm volatile("cp.async.wait_group 1;" ::: "memory");
          fence_proxy();
          mbar_arrive(smem_u32(full + prev));
        }
        prev = slot;
        if (++slot == kSlotsC) {
          slot = 0;
          phase ^= 1u;
        }
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (prev >= 0) {
      fence_proxy();
      mbar_arrive(smem_u32(full + prev));
    }
  } else if (warp == 0 && lane == 0) {
    // ---------------- products ----------------
    // One thread's instructions are the pace of a block here, so rings are
    // counted, not divided, and every descriptor is a constant away from two.
    constexpr int G = L::kGroups;
    int slot = 0;
    uint32_t phase = 0;
    int fresh = 0;            // group of the next output plane to open
    uint32_t fresh_phase = 1; // parity its drained barrier is waited for
    int done = 0;             // group of the next output plane to finish
    bool ok = true, issued = false;
    const uint32_t idesc0 = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kTileM >> 4) << 24);
    for (int t = blockIdx.x; ok && t < P.items; t += gridDim.x) {
      const March m = march_of(P, t);
      const int p1 = min(m.z1 + 1, P.Z - 1);
      int ga = fresh;     // group of the lowest output plane in the window
      int opened = m.z0;  // the next output plane to open
      for (int p = max(m.z0 - 1, 0); p <= p1; p++) {
        const int za = max(p - 1, m.z0), zb = min(p + 1, m.z1);  // output planes of this one
        if (p - 1 > m.z0) ga = ga + 1 == G ? 0 : ga + 1;
        while (ok && opened <= zb) {  // groups entering the window are drained and zero
          ok = mbar_wait(smem_u32(acc_empty + fresh), fresh_phase, abort_flag, P.err);
          opened++;
          if (++fresh == G) {
            fresh = 0;
            fresh_phase ^= 1u;
          }
        }
        if (!ok || !mbar_wait(smem_u32(full + slot), phase, abort_flag, P.err)) {
          ok = false;
          break;
        }
        fence_after();
        const int cnt = zb - za + 1;
        const int n1 = min(cnt, G - ga), n2 = cnt - n1;  // groups up to the ring's end, and after
        const uint32_t d1 = tmem + (uint32_t)(ga * NCH);
        const uint32_t i1 = idesc0 | ((uint32_t)(n1 * NCH >> 3) << 17);
        const uint64_t a0 =
            smem_desc_plain(planes + (uint32_t)slot * L::kSlotB, kGroupB, kRowB);
        const uint64_t b0 = smem_desc_plain(
            weights + (uint32_t)((za - (p - 1)) * NCH * 16), 3 * NCH * 16, 128);
        const auto a_at = [](int q, int j) {
          return (uint64_t)((j * 2 * kGroupB + q / 3 * kRowB + q % 3 * 16) >> 4);
        };
        const auto b_at = [](int q, int j) {
          return (uint64_t)((q * (int)L::kTapB + j * 2 * 3 * NCH * 16) >> 4);
        };
        if (n2 == 0) {
#pragma unroll
          for (int q = 0; q < 9; q++)
#pragma unroll
            for (int j = 0; j < CIN / 16; j++)
              mma_f16(d1, a0 + a_at(q, j), b0 + b_at(q, j), i1, 1u);
        } else {
          const uint32_t i2 = idesc0 | ((uint32_t)(n2 * NCH >> 3) << 17);
          const uint64_t b2 = b0 + (uint64_t)(n1 * NCH);
#pragma unroll
          for (int q = 0; q < 9; q++)
#pragma unroll
            for (int j = 0; j < CIN / 16; j++) {
              mma_f16(d1, a0 + a_at(q, j), b0 + b_at(q, j), i1, 1u);
              mma_f16(tmem, a0 + a_at(q, j), b2 + b_at(q, j), i2, 1u);
            }
        }
        issued = true;
        mma_commit(smem_u32(empty + slot));
        for (int z = max(p - 1, m.z0); z <= (p == p1 ? m.z1 : p - 1); z++) {
          mma_commit(smem_u32(acc_full + done));
          if (++done == G) done = 0;
        }
        if (++slot == kSlotsC) {
          slot = 0;
          phase ^= 1u;
        }
      }
    }
    if (!ok && issued) {
      // wait for every product already issued, on a barrier that nothing else completes now
      mma_commit(smem_u32(empty + slot));
      mbar_drain(smem_u32(empty + slot), phase);
    }
  } else if (warp >= 4) {
    // ---------------- epilogue: tensor memory -> bias, ReLU -> global ----------------
    const int q = warp & 3, row = 32 * q + lane;  // accumulator row: 8 y + x in the column
    int g = L::kGroups - 1;
    uint32_t phase = 1;
    bool ok = true;
    for (int t = blockIdx.x; ok && t < P.items; t += gridDim.x) {
      const March m = march_of(P, t);
      const int x = m.x0 + (row & 7), y = m.y0 + (row >> 3);
      const bool in = x < P.X && y < P.Y;
      for (int z = m.z0; z <= m.z1; z++) {
        if (++g == L::kGroups) {
          g = 0;
          phase ^= 1u;
        }
        const bool ready = mbar_wait(smem_u32(acc_full + g), phase, abort_flag, P.err);
        if (!__all_sync(0xffffffffu, ready)) {
          ok = false;
          break;
        }
        fence_after();
        const uint32_t addr = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(g * NCH);
        float v[NCH];
#pragma unroll
        for (int c = 0; c < NCH; c += 16) {
          float part[16];
          tmem_ld16(addr + (uint32_t)c, part);
#pragma unroll
          for (int e = 0; e < 16; e++) v[c + e] = part[e];
        }
        tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < NCH; c += 16) tmem_zero16(addr + (uint32_t)c);
        tmem_wait_st();
        fence_before();
        mbar_arrive(smem_u32(acc_empty + g));
        if (!in) continue;
        const int64_t cell = (((int64_t)m.b * P.Z + z) * P.Y + y) * P.X + x;
        if (P.kind == TC_ONE) {  // the output layer, its weights padded to 16 rows
          const float r = v[0] + (P.bias ? __ldg(P.bias) : 0.0f);
          static_cast<float *>(P.out)[cell] = P.relu ? fmaxf(r, 0.0f) : r;
          continue;
        }
        if (P.bias) {
#pragma unroll
          for (int c = 0; c < NCH; c++) v[c] += __ldg(P.bias + c);
        }
        if (P.relu) {
#pragma unroll
          for (int c = 0; c < NCH; c++) v[c] = fmaxf(v[c], 0.0f);
        }
        if (P.kind == TC_MASKED) {
          const uint4 *k = reinterpret_cast<const uint4 *>(P.mask + cell * NCH);
#pragma unroll
          for (int c = 0; c < NCH; c += 8) {
            const uint4 w = __ldg(k + c / 8);
            const uint32_t u[4] = { w.x, w.y, w.z, w.w };
#pragma unroll
            for (int e = 0; e < 8; e++) {  // as floats: BF16 is the upper half
              const float f = __uint_as_float(e & 1 ? u[e / 2] & 0xffff0000u : u[e / 2] << 16);
              v[c + e] = f > 0.0f ? v[c + e] : 0.0f;
            }
          }
        }
        if (P.kind == TC_BF16 || P.kind == TC_MASKED) {
          uint4 *o = reinterpret_cast<uint4 *>(static_cast<__nv_bfloat16 *>(P.out) + cell * NCH);
#pragma unroll
          for (int c = 0; c < NCH; c += 8)
            o[c / 8] = make_uint4(pack2(v[c], v[c + 1]), pack2(v[c + 2], v[c + 3]),
                pack2(v[c + 4], v[c + 5]), pack2(v[c + 6], v[c + 7]));
        } else {
          const bool split = P.kind == TC_SPLIT;
          float4 *o = reinterpret_cast<float4 *>(static_cast<float *>(P.out) + cell * (split ? 32 : NCH));
          float4 *o2 = reinterpret_cast<float4 *>(static_cast<float *>(P.out2) + cell * 16) - 8;
#pragma unroll
          for (int c = 0; c < NCH; c += 4)
            (split && c >= 32 ? o2 : o)[c / 4] = make_float4(v[c], v[c + 1], v[c + 2], v[c + 3]);
        }
      }
    }
  }
  fence_before();
  __syncthreads();
  if (warp == 0) {
    __syncwarp();
    fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(L::kCols)
                 : "memory");
  }
}

// ------------------------------------------------------------------ host side

PFN_cuTensorMapEncodeTiled_v12000 encode_fn()
{
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
            &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }
  return fn;
}

CUtensorMapSwizzle swizzle_for(int channels)
{
  return channels == 64 ? CU_TENSOR_MAP_SWIZZLE_128B
                        : channels == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B;
}

// channels-last BF16 volume [zb][y][x][C] as a 4-D map (C, Y, X, Z*B) -- y
// before x, so a box (C, 8, 18, 1) lands as 18 x-columns of 8 cell rows --
// one C x 2-byte row per cell, swizzled over that span
bool map_volume(CUtensorMap *m, const void *base, int C, int X, int Y, int ZB)
{
  auto fn = encode_fn();
  if (!fn) {
    fail(NUSIF_ERR_CUDA, "unet: cuTensorMapEncodeTiled unavailable");
    return false;
  }
  const cuuint64_t dims[4] = { (cuuint64_t)C, (cuuint64_t)Y, (cuuint64_t)X, (cuuint64_t)ZB };
  const cuuint64_t strides[3] = { (cuuint64_t)X * C * 2, (cuuint64_t)C * 2,
    (cuuint64_t)Y * X * C * 2 };
  const cuuint32_t box[4] = { (cuuint32_t)C, (cuuint32_t)kTileY, (cuuint32_t)kBoxX, 1 };
  const cuuint32_t es[4] = { 1, 1, 1, 1 };
  const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void *>(base), dims,
      strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_for(C),
      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    fail(NUSIF_ERR_CUDA, "unet: tensor map of a %dx%dx%dx%d volume failed (%d)", C, X, Y, ZB, (int)r);
    return false;
  }
  return true;
}

// weights [27][N][K] as a 3-D map (K, N, 27), box (C, N, 3): the C columns of
// one source for one (dz, dy) row of three taps, swizzled like that source's
// cell rows
bool map_weights(CUtensorMap *m, const void *base, int K, int N, int C)
{
  auto fn = encode_fn();
  if (!fn) {
    fail(NUSIF_ERR_CUDA, "unet: cuTensorMapEncodeTiled unavailable");
    return false;
  }
  const cuuint64_t dims[3] = { (cuuint64_t)K, (cuuint64_t)N, 27 };
  const cuuint64_t strides[2] = { (cuuint64_t)K * 2, (cuuint64_t)N * K * 2 };
  const cuuint32_t box[3] = { (cuuint32_t)C, (cuuint32_t)N, 3 };
  const cuuint32_t es[3] = { 1, 1, 1 };
  const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void *>(base), dims,
      strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_for(C),
      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    fail(NUSIF_ERR_CUDA, "unet: weight tensor map %dx%d failed (%d)", K, N, (int)r);
    return false;
  }
  return true;
}

int sm_count_tc()
{
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 152;
  }
  return n;
}

uint32_t align1k(uint32_t x) { return (x + 1023u) & ~1023u; }

template <int NCH>
bool launch_tc(const CUtensorMap &a0, const CUtensorMap &a1, const CUtensorMap &w0,
    const CUtensorMap &w1, TcParams P)
{
  // per source: the box of 18 x-columns (8 cell rows each), then the row's
  // three taps' weights [3][N][C], each region 1024-byte aligned (the
  // 128-byte swizzle's atom; an x-column and a tap's weights are whole
  // multiples of every swizzle's 8-row repeat)
  uint32_t off = 0, tx = 0;
  for (int src = 0; src < 2; src++) {
    const uint32_t rb = 2u * (uint32_t)(src == 0 ? P.C0 : P.C1);
    P.atom[src] = (uint32_t)kTileY * rb;
    P.wtap[src] = (uint32_t)NCH * rb;
    P.a_off[src] = off;
    off = align1k(off + (uint32_t)kBoxX * P.atom[src]);
    P.b_off[src] = off;
    off = align1k(off + 3u * P.wtap[src]);
    if (src == 0 || P.C1 > 0) tx += (uint32_t)kBoxX * P.atom[src] + 3u * P.wtap[src];
  }
  P.stage_bytes = off;
  P.tx_bytes = tx;
  const size_t stage_bytes = P.stage_bytes;
  // two stages: the fewer the stages, the more blocks an SM holds, and more
  // blocks measured faster than deeper pipelines; NUSIF_TC_STAGES overrides the
  // count
  int stages = 2;
  if (const char *e = getenv("NUSIF_TC_STAGES")) {
    const int s = atoi(e);
    if (s >= 2) stages = s;
  }
  const int fit = (int)((227 * 1024 - kBarBytes - 1024) / stage_bytes);
  if (stages > fit) stages = fit;
  if (stages > kMaxStages) stages = kMaxStages;
  if (stages < 2) stages = 2;
  P.stages = stages;
  int cols = 32;
  while (cols < 2 * NCH) cols <<= 1;
  P.tmem_cols = cols;
  // barriers and flags, alignment to 1024 bytes, stages
  const size_t smem = kBarBytes + 1024 + (size_t)stages * stage_bytes;
  if (smem > 227 * 1024) {
    fail(NUSIF_ERR_ARG, "unet: convolution stage of %zu bytes too large", stage_bytes);
    return false;
  }
  // at most 512 / cols blocks of an SM may hold tensor memory at once
  const int per_sm_tmem = 512 / cols;
  static bool attr_set[64] = {};
  int dev = 0;
  if (!cuda_ok(cudaGetDevice(&dev), "cudaGetDevice")) return false;
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    if (!cuda_ok(cudaFuncSetAttribute(k_conv_tc<NCH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                     227 * 1024),
            "k_conv_tc shared memory"))
      return false;
    attr_set[dev] = true;
  }
  // a persistent grid: no more blocks than can be resident at once, by shared
  // memory (1 KB reserved per block), registers (8-register granules per
  // thread) and tensor memory
  cudaFuncAttributes fa{};
  if (!cuda_ok(cudaFuncGetAttributes(&fa, k_conv_tc<NCH>), "k_conv_tc attributes")) return false;
  const int regs_block = ((fa.numRegs + 7) / 8) * 8 * kThreads;
  int per_sm = (int)((228 * 1024) / (smem + 1024));
  if (regs_block > 0 && per_sm > 65536 / regs_block) per_sm = 65536 / regs_block;
  if (per_sm > per_sm_tmem) per_sm = per_sm_tmem;
  if (per_sm < 1) per_sm = 1;
  int grid = sm_count_tc() * per_sm;
  if (grid > P.ntiles) grid = P.ntiles;
  P.idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NCH >> 3) << 17) |
            ((uint32_t)(kTileM >> 4) << 24);
  k_conv_tc<NCH><<<grid, kThreads, smem, stream()>>>(a0, a1, w0, w1, P);
  return launched("k_conv_tc");
}

template <int NCH, int CIN>
bool launch_col(ColParams P)
{
  using L = Col<NCH, CIN>;
  static bool attr_set[64] = {};
  int dev = 0;
  if (!cuda_ok(cudaGetDevice(&dev), "cudaGetDevice")) return false;
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    if (!cuda_ok(cudaFuncSetAttribute(k_conv_col<NCH, CIN>,
                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::kSmem),
            "k_conv_col shared memory"))
      return false;
    attr_set[dev] = true;
  }
  // a persistent grid: no more blocks than can be resident at once, by shared
  // memory (1 KB reserved per block), registers and tensor memory
  static int regs = 0;
  if (regs == 0) {
    cudaFuncAttributes fa{};
    if (!cuda_ok(cudaFuncGetAttributes(&fa, k_conv_col<NCH, CIN>), "k_conv_col attributes"))
      return false;
    regs = ((fa.numRegs + 7) / 8) * 8 * kColThreads;
  }
  int per_sm = (int)((228 * 1024) / (L::kSmem + 1024));
  if (per_sm > 65536 / regs) per_sm = 65536 / regs;
  if (per_sm > 512 / L::kCols) per_sm = 512 / L::kCols;
  if (per_sm < 1) per_sm = 1;
  const int wave = sm_count_tc() * per_sm;
  // planes of a march: the least (marches of the busiest block) x (planes + 2
  // read around them)
  const int64_t columns = (int64_t)P.B * P.tx * P.ty;
  int64_t best = -1;
  for (int zl = 1; zl <= P.Z; zl++) {
    const int64_t n = columns * ((P.Z + zl - 1) / zl);
    const int64_t cost = ((n + wave - 1) / wave) * (zl + 2);
    if (best < 0 || cost < best) {
      best = cost;
      P.zl = zl;
    }
  }
  P.zt = (P.Z + P.zl - 1) / P.zl;
  P.items = (int)(columns * P.zt);
  const int grid = P.items < wave ? P.items : wave;
  k_conv_col<NCH, CIN><<<grid, kColThreads, L::kSmem, stream()>>>(P);
  return launched("k_conv_col");
}

// the layers of the marching form, as 100 N + channels in: at most 48 channels
// on either side (the weights of all taps and four planes fit shared memory
// several blocks at a time)
bool col_layer(int N, int C)
{
  switch (100 * N + C) {
  case 1616: case 1632: case 1648: case 3216: case 3232: case 4816: return true;
  }
  return false;
}

}  // namespace

bool tc_conv_supported(int X, int Y, int Z, int B, int N, int C0, int C1)
{
  if (X <= 0 || Y <= 0 || Z <= 0 || B <= 0) return false;
  auto ok_c = [](int c) { return c == 16 || c == 32 || c == 64; };
  if (!ok_c(C0) || (C1 != 0 && !ok_c(C1))) return false;
  if (!col_layer(N, C0 + C1) && N != 32 && N != 64 && N != 96) return false;
  if (X % kTileX || Y % kTileY) return false;
  return encode_fn() != nullptr;
}

bool tc_conv_marches(int N, int C) { return col_layer(N, C); }

bool tc_conv(const void *s0, int C0, const void *s1, int C1, int B, int Z, int Y, int X,
    const void *w, int N, const float *bias, int relu, TcOut kind, void *out, int *err, int up0,
    const void *mask, void *out2)
{
  if (col_layer(N, C0 + C1)) {
    ColParams c{};
    c.s0 = static_cast<const __nv_bfloat16 *>(s0);
    c.s1 = static_cast<const __nv_bfloat16 *>(s1);
    c.w = static_cast<const __nv_bfloat16 *>(w);
    c.C0 = C0;
    c.C1 = C1;
    c.up0 = up0;
    c.X = X;
    c.Y = Y;
    c.Z = Z;
    c.B = B;
    c.tx = (X + kColX - 1) / kColX;
    c.ty = (Y + kColY - 1) / kColY;
    c.bias = bias;
    c.relu = relu;
    c.kind = (int)kind;
    c.out = out;
    c.out2 = out2;
    c.mask = static_cast<const __nv_bfloat16 *>(mask);
    c.err = err;
    switch (100 * N + C0 + C1) {
    case 1616: return launch_col<16, 16>(c);
    case 1632: return launch_col<16, 32>(c);
    case 1648: return launch_col<16, 48>(c);
    case 3216: return launch_col<32, 16>(c);
    case 3232: return launch_col<32, 32>(c);
    default: return launch_col<48, 16>(c);
    }
  }
  if (up0 || (kind != TC_BF16 && kind != TC_F32)) {
    fail(NUSIF_ERR_ARG, "unet: a form of convolution that %d -> %d channels has not", C0 + C1, N);
    return false;
  }
  TcParams P{};
  P.N = N;
  P.C0 = C0;
  P.C1 = C1;
  P.X = X;
  P.Y = Y;
  P.Z = Z;
  P.B = B;
  P.tx = X / kTileX;
  P.ty = Y / kTileY;
  P.ntiles = (int)((int64_t)B * Z * P.ty * P.tx);
  P.bias = bias;
  P.relu = relu;
  P.out_bf16 = kind == TC_BF16 ? 1 : 0;
  P.out = out;
  P.err = err;
  CUtensorMap a0, a1, w0, w1;
  if (!map_volume(&a0, s0, C0, X, Y, Z * B)) return false;
  if (!map_weights(&w0, w, C0 + C1, N, C0)) return false;
  if (C1 > 0) {
    if (!map_volume(&a1, s1, C1, X, Y, Z * B)) return false;
    if (!map_weights(&w1, w, C0 + C1, N, C1)) return false;
  } else {
    a1 = a0;
    w1 = w0;
  }
  switch (N) {
  case 32: return launch_tc<32>(a0, a1, w0, w1, P);
  case 64: return launch_tc<64>(a0, a1, w0, w1, P);
  case 96: return launch_tc<96>(a0, a1, w0, w1, P);
  }
  fail(NUSIF_ERR_ARG, "unet: no tensor-core convolution for %d output channels", N);
  return false;
}

}  // namespace nusif
