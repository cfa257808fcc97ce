// Red-black SOR, iterations 2 and on, as whole-iteration sweeps on the change
// of p (src/solver-rb.c:50-151 semantics; the first iteration runs on p
// itself, k_sor_pass in solver.cu).
//
// The scheme is linear: with P the pressure after some iterations (whose
// ghosts then equal the cells beside them) and p = P + d, an iteration relaxes
// d against r0 = rhs - A P, formed in FP64, and the residual is the
// same. d and r0 are kept as pairs of FP32 numbers (df32.cuh; plain doubles
// with arith fp64), so an update needs no split of binary64 operands and no
// FP64 instruction, and its rounding scales with |d|, not |p|. P is the
// pressure after the first iteration, then, every few (next_fold), P + d in
// binary64, and so is p at the end: the error of a solve against 64 bits is below
// that of the scheme on p itself, wherever it starts. The factors
// are folded into the constants: an update is c + D with
//   D = -factor r = f_x (w + e - 2 c) + f_y (s + n - 2 c) + f_z (b + t - 2 c) - factor r0,
// and the sum of r^2 is that of D^2 over factor^2. factor is omega h^2 / 6, of
// any size, so d and r0 are kept times the power of two that brings it to 1 or
// more: D^2 is then of the size of r^2, and the range in which pairs hold it
// does not depend on the cells' size.
//
// Layout: d and r0 with the colours apart, [colour][k][j][t], t the pair
// (2t, 2t+1) of a row, so a thread's loads and stores are contiguous over the
// warp whatever colour it works on. Indices are 0-based here; the first
// colour ((i + j + k) odd, 1-based) has an even 0-based sum.
//
// One kernel is one iteration, exact: it reads d, writes the other copy, so
// no block reads what another writes. A thread owns one pair of columns and
// marches over A.kb planes: at plane k it relaxes the pair's first-colour
// cell of plane k and then, in the same column, the second-colour cell of
// plane k - 1, whose neighbours are all new by then. z-neighbours and one
// x-neighbour are in its registers; the other x- and both y-neighbours come
// from half planes (one colour) in shared memory: eight 8-byte accesses for
// two updates and one barrier per plane. The tile's rows are surrounded by
// one row (and pair, where x is tiled) that only relaxes the first colour,
// again by its owner: blocks are independent.
//
// Walls: the stale ghost of the reference is the wall cell's old value. d has
// a ghost row and plane on each side; they hold the wall's cells with the
// colours exchanged, which puts a wall cell's old value where each of its
// neighbours looks, and so does the missing second column of an odd row's
// last pair. In x the wall is a select.
//
// The stop test costs no tail: block sums of D^2 go to part_out, and every
// block of the next iteration's kernel folds them, in one order, while its
// first planes load, then decides alike (k_rb_fold first where there are
// many). R_m, the carried residual after m iterations, is kept in res[m & 1]:
// kernel n reads R_(n-2) and iteration n - 1's sums, block 0 stores R_(n-1).
// Sums stay pairs of FP32 numbers to the end (doubles with arith fp64): an FP64
// addition costs a warp 16 cycles of GB300's FP64 pipe and about 100 of latency
// (block sums and fold in FP64: 64^3 5.6 -> 6.2 us an iteration). So that the
// sum over a grid keeps the range of a cell's square, a thread's sum is taken
// times 2^-30, or less where eps^2 would come near the smallest float.
//
// What bounds it: at 128^3 instruction issue (about 215 thread instructions per
// cell, ring included; k_sor_pass in two launches about 520), at 64^3 half
// issue, half the launch and its first loads (about 3 us). An iteration of a
// solve, two launches of k_sor_pass -> one sweep and its share of the folds:
// 128^3 47 -> 20.6 us, 64^3 19.7 -> 7.0, 200 x 40 x 40 28.9 -> 8.3, and the error
// against 64 bits 1.4e-14 -> 1.3e-16, 1.1e-14 -> 1e-16, 2.9e-13 -> 5e-16. One
// cooperative kernel for all iterations, its blocks exchanging sums through L2,
// took 2 us more per iteration than launches (two device-wide fences); letting
// the next kernel's blocks in early took 1 us more (they double up on the idle
// SMs).
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <utility>
#include <type_traits>

#include "df32.cuh"
#include "nusif_internal.h"
#include "reduce.cuh"
#include "solver_internal.h"

namespace nusif {
namespace {

constexpr int kMaxThreads = 640;

// factor / h^2 of each axis
template <typename V>
struct Consts {
  V fx, fy, fz;
};
Consts<df::f2> consts(const SorArgs &A, df::f2)
{
  return { df::from_double_rn(A.factor * A.idx2), df::from_double_rn(A.factor * A.idy2),
           df::from_double_rn(A.factor * A.idz2) };
}
Consts<double> consts(const SorArgs &A, double)
{
  return { A.factor * A.idx2, A.factor * A.idy2, A.factor * A.idz2 };
}

// Each factor is rounded by itself, so a small one (a long spacing among short
// ones) keeps its bits.

// a - K c, an unnormalised pair
template <int K>
__device__ __forceinline__ df::f2 minus(df::f2 a, df::f2 c)
{
  using namespace df;
  const f2 p = two_prod((float)-K, c.hi);  // (exact: no low part where K is a power of two)
  const f2 s = two_sum(p.hi, a.hi);
  const float lo = fmaf_((float)-K, c.lo, a.lo);
  return f2{ s.hi, K == 2 ? add_(s.lo, lo) : add_(add_(s.lo, p.lo), lo) };
}

// the change D of a cell c with the neighbours w, e, s, n, b, t; r = -factor
// r0. A constant d has no change, whatever the factors: the cell is taken from
// its neighbours before the product. (With a factor of its own the cell's
// product rounds at the size of d, in the same direction every iteration.)
// CUBE: one spacing on all axes, one product instead of three. What comes from
// registers (b, t) first. With factors of a common quantum, whose sum the
// cell's factor was exactly, 64 x 64 x 4 cells of a 0.01 x 1 x 1 box from rest,
// 500 iterations, were 8.3e-13 (fp64 4.6e-13) off, here 1.2e-13 (4.2e-15), on p
// itself 3.4e-13 (7.0e-15); pairs of unlike spacings take 5 to 10% more time.
template <bool CUBE>
__device__ __forceinline__ df::f2 change(const Consts<df::f2> &C, df::f2 c, df::f2 w, df::f2 e,
    df::f2 s, df::f2 n, df::f2 b, df::f2 t, df::f2 r)
{
  using namespace df;
  f2 v;
  if (CUBE) {
    v = add_u(add_u(add_u(w, e), add_u(s, n)), minus<6>(add_u(b, t), c));
    v = fma_u(v, C.fx, r);
  } else {
    v = fma_u(minus<2>(add_u(b, t), c), C.fz, r);
    v = fma_u(minus<2>(add_u(s, n), c), C.fy, v);
    v = fma_u(minus<2>(add_u(w, e), c), C.fx, v);
  }
  return renorm(v.hi, v.lo);
}
template <bool CUBE>
__device__ __forceinline__ double change(const Consts<double> &C, double c, double w, double e,
    double s, double n, double b, double t, double r)
{
  if (CUBE) return ::fma(((w + e) + (s + n)) + ::fma(-6.0, c, b + t), C.fx, r);
  double v = ::fma(::fma(-2.0, c, b + t), C.fz, r);
  v = ::fma(::fma(-2.0, c, s + n), C.fy, v);
  return ::fma(::fma(-2.0, c, w + e), C.fx, v);
}
__device__ __forceinline__ df::f2 moved(df::f2 c, df::f2 D) { return df::add(c, D); }
__device__ __forceinline__ double moved(double c, double D) { return c + D; }
__device__ __forceinline__ void add_square(df::f2 &acc, df::f2 D)
{
  acc = df::add_u(acc, df::mul_u(D, D));
}
__device__ __forceinline__ void add_square(double &acc, double D) { acc = ::fma(D, D, acc); }
__device__ __forceinline__ df::f2 to_cell(double x, df::f2) { return df::split(x); }
__device__ __forceinline__ double to_cell(double x, double) { return x; }
// p + d, d kept times 1 / unit (the products are exact)
__device__ __forceinline__ double plus(double p, df::f2 d, double unit)
{
  return ::fma(df::widen(d.lo), unit, ::fma(df::widen(d.hi), unit, p));
}
__device__ __forceinline__ double plus(double p, double d, double unit) { return ::fma(d, unit, p); }

struct SweepArgs {
  int nx, ny, nz, np;  // np: pairs per row
  int pitch;           // cells of one colour's plane: np * (ny + 2)
  int half;            // cells of one colour's array: pitch * (nz + 4), planes -2 .. nz + 1
  int own, halo;       // pairs a block owns per row; 1 where x is tiled
  int rows;            // rows a block owns
  int kb;              // planes a block owns
  // offset of pair T of row j (-1 .. ny) of plane k (-2 .. nz + 1)
  __host__ __device__ __forceinline__ int at(int T, int j, int k) const
  {
    return (k + 2) * pitch + (j + 1) * np + T;
  }
};

__device__ __forceinline__ df::f2 join(df::f2 a, df::f2 b) { return df::add(a, b); }
__device__ __forceinline__ double join(double a, double b) { return a + b; }
__device__ __forceinline__ df::f2 from_lane(df::f2 v, int o)
{
  return df::f2{ __shfl_xor_sync(0xffffffffu, v.hi, o), __shfl_xor_sync(0xffffffffu, v.lo, o) };
}
__device__ __forceinline__ double from_lane(double v, int o)
{
  return __shfl_xor_sync(0xffffffffu, v, o);
}
template <typename V>
__device__ __forceinline__ V warp_total(V v)
{
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = join(v, from_lane(v, o));
  return v;
}

__device__ __forceinline__ df::f2 load_sum(const df::f2 *p)
{
  const float2 x = __ldcg(reinterpret_cast<const float2 *>(p));
  return df::f2{ x.x, x.y };
}
__device__ __forceinline__ double load_sum(const double *p) { return __ldcg(p); }

// one warp's sum of a list, in a fixed order
template <typename V>
__device__ __forceinline__ V fold_list(const V *part, int np, int lane)
{
  constexpr int kAtOnce = 5;  // loads in flight
  V v{};
  for (int q0 = lane; q0 < np; q0 += 32 * kAtOnce) {
    V x[kAtOnce];
#pragma unroll
    for (int u = 0; u < kAtOnce; u++) x[u] = load_sum(part + min(q0 + 32 * u, np - 1));
#pragma unroll
    for (int u = 0; u < kAtOnce; u++)
      if (q0 + 32 * u < np) v = join(v, x[u]);
  }
  return warp_total(v);
}

__device__ __forceinline__ double as_double(df::f2 v) { return df::to_double(v); }
__device__ __forceinline__ double as_double(double v) { return v; }
// a thread's sum of squares, to be added to others'
__device__ __forceinline__ df::f2 scaled(df::f2 a, float k) { return df::renorm(a.hi * k, a.lo * k); }
__device__ __forceinline__ double scaled(double a, float) { return a; }

__device__ __forceinline__ bool is_done(const RbState *st)
{
  return *reinterpret_cast<const volatile int *>(&st->s.done) != 0;
}

// the carried residual after an iteration whose D^2 sum to `sum`
template <typename V>
__device__ __forceinline__ double carried(const RbState *st, double before, V sum)
{
  return (before + as_double(sum) * st->inv_factor2) * st->inv_ncell;
}

// a pair's cell in one column: the new first-colour value two planes below
// the one it is relaxed in next, and the old second-colour value one below
template <typename V>
struct Window {
  V nf, o;
};
// what a step reads from memory: first colour of plane k, second of k + 1, and
// r of the first colour of k and of the second of k - 1; the ring rows' outer
// neighbour
template <typename V>
struct Ahead {
  V f, s, rf, rs, e;
};

// iteration n, with the np sums of the previous one in part_in (np 0: that one
// ran on p itself); down: the scale of the sums
template <typename V, bool CUBE>
__global__ void __launch_bounds__(kMaxThreads) k_rb_sweep(SweepArgs A, Consts<V> C,
    const V *d, V *dout, const V *r0, RbState *st, const V *part_in, V *part_out, int n, int np,
    float down)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ V sm[kMaxThreads / 32];
  __shared__ int go_on;
  const int pw = A.own + 2 * A.halo, nrow = A.rows + 2;
  const int plane_n = pw * nrow, plane_o = pw * (nrow + 2);
  // old second colour of plane k (rows j0 - 2 .. j0 + rows + 1), new first
  // colour of plane k (one row less on each side), two planes each
  V *const olds = reinterpret_cast<V *>(smem_raw);
  V *const news = olds + 2 * plane_o;
  const int tid = threadIdx.x, lane = tid & 31;
  const bool live = tid < plane_n;
  const int row = min(tid / pw, nrow - 1), t = tid - (tid / pw) * pw;
  const int T = (int)blockIdx.x * A.own + t - A.halo;  // the pair
  const int j = (int)blockIdx.y * A.rows + row - 1;
  const int k0 = blockIdx.z * A.kb, k1 = min(k0 + A.kb, A.nz) - 1;
  const int nx = A.nx, ny = A.ny, nz = A.nz, pitch = A.pitch, half = A.half;
  const int bid = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
  const bool cell_in = live && T >= 0 && T < A.np && j >= 0 && j < ny;
  const bool own = cell_in && t >= A.halo && t < A.halo + A.own && row >= 1 && row <= A.rows;
  const bool lower = row == 0, upper = row == nrow - 1, ring = live && (lower || upper);
  // loads stay in the array: pairs in the row, rows up to the ghost rows
  const int Tc = min(max(T, 0), A.np - 1);
  const int base = A.at(Tc, min(j, ny), k0 - 1);  // plane k0 - 1
  const int base_e = A.at(Tc, min(max(lower ? j - 1 : j + 1, -1), ny), k0 - 1) + half;

  // step q = k - (k0 - 1); window X is the column relaxed in even steps
  const int colx = (j + k0 - 1) & 1;
  const auto wall = [&](int col) { return col == 0 ? T == 0 : 2 * T + 1 >= nx - 1; };
  const bool wall_x = wall(colx), wall_y = wall(1 - colx);
  const bool lone = 2 * T + 1 >= nx;  // odd nx: the last pair has no second column
  const bool valid_x = cell_in && !(lone && colx == 1), valid_y = cell_in && !(lone && colx == 0);
  // shared-memory offsets: own cell, and the x-neighbour outside the pair
  const int so = (row + 1) * pw + t, sf = row * pw + t;
  const int dl = t > 0 ? -1 : 0, dr = t < pw - 1 ? 1 : 0;
  const int ax = colx ? dr : dl, ay = colx ? dl : dr;
  const int s_ring = lower ? t : (nrow + 1) * pw + t;

  // everything read from here on is the previous kernel's work; all of it is
  // asked for at once
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const bool over = is_done(st);
  int o = base;  // plane k's offset
  Window<V> X, Y;
  Ahead<V> a0, a1;  // of even and odd steps
  X.o = d[base + half - pitch];
  Y.o = d[base + half];
  a0.f = d[base];
  a0.s = d[base + half + pitch];
  a0.rf = r0[base];
  a1.f = d[base + pitch];
  a1.s = d[base + half + 2 * pitch];
  a1.rf = r0[base + pitch];
  a1.rs = r0[base + half];
  a0.rs = a1.rs;
  a0.e = a1.e = a0.f;
  if (ring) {
    a0.e = d[base_e];
    a1.e = d[base_e + pitch];
  }
  X.nf = Y.nf = X.o;  // not used before they are set
  if (tid < 32) {
    // the previous iteration's residual, and whether this one runs
    const double before = __ldcg(&st->res[n & 1]), first = __ldcg(&st->s.res);
    const double epssq = __ldcg(&st->s.epssq);
    const int itermax = __ldcg(&st->s.itermax);
    bool go = true;
    if (np > 0) {
      const V sum = fold_list(part_in, np, lane);
      if (lane == 0) {
        const double res = carried(st, before, sum);
        go = res >= epssq && n - 1 < itermax;
        if (bid == 0 && !over) {
          st->res[(n - 1) & 1] = res;
          if (!go) {
            st->s.res = res;
            st->s.it = n - 1;
            st->s.done = 1;
          }
        }
      }
    } else if (bid == 0 && lane == 0) {
      st->res[(n - 1) & 1] = first;
    }
    if (lane == 0) go_on = go && !over;
  }
  __syncthreads();
  if (!go_on) return;

  V acc{};
  // P: the window relaxed in this step, Q: the other one
  const auto step = [&](int k, Window<V> &P, Window<V> &Q, Ahead<V> &a, int buf, bool wallP,
                        bool validP, int adj) {
    V *const so_k = olds + buf * plane_o + so, *const nf_k = news + buf * plane_n + sf;
    const V *const nf_m = news + (buf ^ 1) * plane_n + sf;
    if (live) so_k[0] = Q.o;
    if (ring) olds[buf * plane_o + s_ring] = a.e;
    const V fc = a.f, sup = a.s, rf = a.rf, rs = a.rs;
    if (k + 2 <= k1 + 1) {
      a.f = d[o + 2 * pitch];
      a.s = d[o + 3 * pitch + half];
      a.rf = r0[o + 2 * pitch];
      a.rs = r0[o + pitch + half];
      if (ring) a.e = d[base_e + (o - base) + 2 * pitch];
    }
    __syncthreads();
    // first colour of plane k
    V nw = fc;
    {
      V x1 = so_k[adj];
      if (wallP) x1 = fc;
      const V D = change<CUBE>(C, fc, x1, Q.o, so_k[-pw], so_k[pw], P.o, sup, rf);
      if (validP && k >= 0 && k < nz) {
        nw = moved(fc, D);
        if (own && k >= k0 && k <= k1) add_square(acc, D);
      }
    }
    if (live) nf_k[0] = nw;
    // second colour of plane k - 1, in the same column
    if (own && k > k0) {
      V x1 = nf_m[adj];
      if (wallP) x1 = P.o;
      V fv = Q.nf, m = P.o;
      const V D = change<CUBE>(C, P.o, x1, Q.nf, nf_m[-pw], nf_m[pw], P.nf, nw, rs);
      if (validP) {
        m = moved(P.o, D);
        add_square(acc, D);
      }
      if (lone) {  // the missing column's entry holds its neighbour's value
        if (validP) fv = m;
        else m = fv;
      }
      V *const w = dout + (o - pitch);
      w[0] = fv;
      w[half] = m;
      if (j == 0) {
        w[half - A.np] = fv;
        w[-A.np] = m;
      }
      if (j == ny - 1) {
        w[half + A.np] = fv;
        w[A.np] = m;
      }
      if (k == 1) {
        w[half - pitch] = fv;
        w[-pitch] = m;
      }
      if (k == nz) {
        w[half + pitch] = fv;
        w[pitch] = m;
      }
    }
    o += pitch;
    P.nf = nw;
    P.o = sup;
  };
  for (int k = k0 - 1; k <= k1 + 1; k += 2) {
    step(k, X, Y, a0, 0, wall_x, valid_x, ax);
    if (k + 1 <= k1 + 1) step(k + 1, Y, X, a1, 1, wall_y, valid_y, ay);
  }
  const V ws = warp_total(scaled(acc, down));
  if (lane == 0) sm[tid >> 5] = ws;
  __syncthreads();
  if (tid < 32) {
    const int nw = blockDim.x >> 5;
    const V sum = warp_total(lane < nw ? sm[lane] : V());
    if (lane == 0) part_out[bid] = sum;
  }
}

// rhs - A P of a cell in FP64, from P's differences: they are near exact where P
// is smooth, where a sum of terms of the size of A P rounds, once for all the
// iterations that follow. CG: past L1, P was written in this kernel.
template <bool CG>
__device__ __forceinline__ double residual_of(const SorArgs &S, const double *p, const double *rhs,
    int c)
{
  const int sj = S.g.sj, sk = S.g.sk;
  const auto ld = [&](int q) { return CG ? __ldcg(p + q) : p[q]; };
  const double m = ld(c);
  double r = rhs[c];
  r = ::fma(-((ld(c - 1) - m) + (ld(c + 1) - m)), S.idx2, r);
  r = ::fma(-((ld(c - sj) - m) + (ld(c + sj) - m)), S.idy2, r);
  return ::fma(-((ld(c - sk) - m) + (ld(c + sk) - m)), S.idz2, r);
}

// a cell's pressure, and the ghosts beside it
__device__ __forceinline__ void store_p(const SweepArgs &A, const Dims &g, double *p, int i, int j,
    int k, double v)
{
  double *c = p + ((k + 1) * g.sk + (j + 1) * g.sj + i + 1);
  *c = v;
  if (i == 0) c[-1] = v;
  if (i == A.nx - 1) c[1] = v;
  if (j == 0) c[-g.sj] = v;
  if (j == A.ny - 1) c[g.sj] = v;
  if (k == 0) c[-g.sk] = v;
  if (k == A.nz - 1) c[g.sk] = v;
}

// p holds n iterations: r0 = -factor (rhs - A P) (S.factor is the scaled one),
// d = 0 with its ghosts (one thread per entry of a colour's array)
template <typename V>
__global__ void __launch_bounds__(256) k_rb_open(SweepArgs A, SorArgs S, const double *__restrict__ p,
    const double *__restrict__ rhs, V *__restrict__ d, V *__restrict__ r0, RbState *st, int n)
{
  if (is_done(st)) return;
  const int q = blockIdx.x * 256 + threadIdx.x;
  if (q == 0) st->base = n;
  if (q >= A.half) return;
  d[q] = d[q + A.half] = V();
  const int T = q % A.np, jk = q / A.np, j = jk % (A.ny + 2) - 1, k = jk / (A.ny + 2) - 2;
  if (j < 0 || j >= A.ny || k < 0 || k >= A.nz) return;
#pragma unroll
  for (int e = 0; e < 2; e++) {
    const int i = 2 * T + e;
    double r = 0.0;
    if (i < A.nx)
      r = residual_of<false>(S, p, rhs, (k + 1) * S.g.sk + (j + 1) * S.g.sj + i + 1);
    r0[((i + j + k) & 1) * A.half + q] = to_cell(-S.factor * r, V());
  }
}

// p = P + d on the cells and the six ghost faces: of iteration n (k_rb_open
// follows), or once the solve is over (n 0)
template <typename V>
__global__ void __launch_bounds__(256) k_rb_close(SweepArgs A, Dims g, double *__restrict__ p,
    const V *__restrict__ d0, const V *__restrict__ d1, double unit, const RbState *st, int n)
{
  if (n > 0 ? is_done(st) : !is_done(st) || st->s.it <= st->base) return;
  const V *d = ((n > 0 ? n : st->s.it) & 1) ? d1 : d0;
  const int q = blockIdx.x * 256 + threadIdx.x;
  if (q >= A.np * A.ny * A.nz) return;
  const int T = q % A.np, jk = q / A.np, j = jk % A.ny, k = jk / A.ny;
#pragma unroll
  for (int e = 0; e < 2; e++) {
    const int i = 2 * T + e;
    if (i >= A.nx) continue;
    const double was = p[(k + 1) * g.sk + (j + 1) * g.sj + i + 1];
    store_p(A, g, p, i, j, k, plus(was, d[((i + j + k) & 1) * A.half + A.at(T, j, k)], unit));
  }
}

// The iterations after which d joins p and r0 is formed anew. Pairs round an
// update at the size of d, and r0's own rounding acts in every iteration alike,
// so d has to stay small against p also where a solve starts far from its end.
// Error against 64 bits after 500 iterations, on p itself | d over the whole solve
// | here (24^3, from a pressure that has nothing to do with the right-hand side):
// pairs 5.3e-14 | 1.3e-12 | 1.1e-14, fp64 6.3e-16 | 8.8e-14 | 3.8e-16; from near
// the end, 6 x 160 x 7 cells of 4 x 1 x 1: pairs 5.1e-13 | 6.1e-14 | 1.9e-15, fp64
// 4.7e-15 | 4.6e-14 | 1.3e-16. (After 8, 32, 128, 512 .. iterations was not
// enough where the right-hand side has a mean: 23^3 ten times the error on p.) A
// fold costs about 75 us at 128^3, where 64 iterations take 1230, and 18 of 430 at
// 64^3.
__host__ __device__ constexpr int next_fold(int n)
{
  return n < 8 ? 8 : n < 32 ? 32 : 32 + 64 * ((n - 32) / 64 + 1);
}

// a long list of block sums folded once instead of by every block of the next sweep
template <typename V>
__global__ void __launch_bounds__(1024) k_rb_fold(const RbState *st, const V *part, int np, V *out)
{
  if (is_done(st)) return;
  __shared__ V sm[32];
  const int t = threadIdx.x;
  V v{};
  for (int q = t; q < np; q += 1024) v = join(v, load_sum(part + q));
  v = warp_total(v);
  if ((t & 31) == 0) sm[t >> 5] = v;
  __syncthreads();
  if (t >= 32) return;
  v = warp_total(sm[t]);
  if (t == 0) *out = v;
}

// after a chunk of sweeps that ended with iteration n: its residual, and
// whether the solve is over (one warp)
template <typename V>
__global__ void k_rb_finish(RbState *st, const V *part, int n, int np)
{
  if (is_done(st)) return;
  const V s = fold_list(part, np, threadIdx.x);
  if (threadIdx.x == 0) {
    const double res = carried(st, st->res[(n - 1) & 1], s);
    st->s.res = res;
    st->s.it = n;
    st->s.done = !(res >= st->s.epssq && n < st->s.itermax);
  }
}

// All the iterations of a small grid in one cluster, d and r0 in shared memory.
// The grid is cut into slabs along its longest axis (2 here, whichever it is of
// x, y and z; 0 is the axis of the pairs), P planes to a block and a copy of the
// neighbours' planes on each side, which they write as they update. Two copies
// of d: an iteration reads one and writes the other, first colour, barrier,
// second colour, barrier. The last warps relax nothing; they sum the squares of
// the iteration before while the others work, send the block's sums to all
// blocks in the first half and decide in the second, so the stop costs one
// iteration too many but no time in each.
//
// What bounds it: the barrier of the cluster (about 0.3 us, twice an iteration)
// and the updates' latency, from 10 thousand cells on their issue on sixteen
// SMs. An iteration, sweeps -> cluster: 12^3 4.9 -> 2.4 us, 20^3 4.4 -> 2.2,
// 64 x 10 x 61 4.4 -> 4.0 (three products per update).
struct ClusterArgs {
  int n[3];       // cells per axis, the slab axis last
  int axis[3];    // which of x, y, z each is
  int np, plane;  // pairs per row and per plane
  int P;          // planes per block
  int blocks;     // of the cluster
  unsigned mrow, mpl;  // 2^32 / np and / plane, rounded up (0: 1)
};

__device__ __forceinline__ void cluster_barrier(int blocks)
{
  if (blocks == 1) {
    __syncthreads();
  } else {
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
  }
}

__device__ __forceinline__ unsigned in_block(const void *p, int rank)
{
  unsigned a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n"
               : "=r"(a)
               : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ void store_in(unsigned at, df::f2 v)
{
  asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};\n" ::"r"(at), "f"(v.hi), "f"(v.lo)
               : "memory");
}
__device__ __forceinline__ void store_in(unsigned at, double v)
{
  asm volatile("st.shared::cluster.f64 [%0], %1;\n" ::"r"(at), "d"(v) : "memory");
}

constexpr int kFoldWarps = 4;
constexpr size_t kClusterSmem = 226 * 1024 - 1024;  // of 227 KB; the kernel has a little of its own

// sums of non-negative pairs that need no order: without renormalising between
__device__ __forceinline__ df::f2 join_u(df::f2 a, df::f2 b) { return df::add_u(a, b); }
__device__ __forceinline__ double join_u(double a, double b) { return a + b; }
template <typename V>
__device__ __forceinline__ V warp_total_u(V v)
{
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = join_u(v, from_lane(v, o));
  return scaled(v, 1.0f);
}

template <typename V, bool CUBE>
__global__ void __launch_bounds__(1024) k_rb_cluster(ClusterArgs A, SweepArgs G, Consts<V> C,
    SorArgs S, double *p, const double *rhs, const V *__restrict__ r0, V *d0, V *d1, double unit,
    RbState *st, float down)
{
  if (is_done(st)) return;  // the same for all blocks
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ V total[16 * kFoldWarps];
  __shared__ int go;
  const int tid = threadIdx.x, lane = tid & 31, workers = blockDim.x - 32 * kFoldWarps;
  const bool work = tid < workers;
  const int rank = blockIdx.x, plane = A.plane, np = A.np;
  const int first = rank * A.P, mine = max(0, min(A.P, A.n[2] - first)) * plane;
  const int size = (A.P + 2) * plane;  // one colour, one copy
  V *const cells = reinterpret_cast<V *>(smem_raw);  // [copy][colour][plane -1 .. P][pair]
  V *const rs = cells + 4 * size;                    // [colour][pair]
  V *const squares = rs + 2 * A.P * plane;           // a worker's sum
  unsigned char *const flag = reinterpret_cast<unsigned char *>(squares + workers);
  const auto cell = [&](int q, int e, int (&x)[3]) {  // of pair q: where it is on the grid
    const int kk = A.mpl ? (int)__umulhi((unsigned)q, A.mpl) : q, jt = q - kk * plane;
    const int j = A.mrow ? (int)__umulhi((unsigned)jt, A.mrow) : jt, t = jt - j * np;
    const int c[3] = { 2 * t + e, j, first + kk };
#pragma unroll
    for (int a = 0; a < 3; a++)
      x[a] = A.axis[0] == a ? c[0] : A.axis[1] == a ? c[1] : c[2];
    return c[0] < A.n[0];
  };
  const auto colour_of = [](const int (&x)[3]) { return (x[0] + x[1] + x[2]) & 1; };
  for (int q = tid; q < 4 * size; q += blockDim.x) cells[q] = V();
  for (int q = tid; q < mine; q += blockDim.x) {
    const int kk = A.mpl ? (int)__umulhi((unsigned)q, A.mpl) : q, jt = q - kk * plane;
    const int j = A.mrow ? (int)__umulhi((unsigned)jt, A.mrow) : jt, t = jt - j * np;
    const int k = first + kk;
    flag[q] = (unsigned char)((t > 0) | (2 * t + 2 < A.n[0]) << 1 | (j > 0) << 2 |
                              (j < A.n[1] - 1) << 3 | (k > 0) << 4 | (k < A.n[2] - 1) << 5 |
                              (2 * t + 1 == A.n[0]) << 6 | ((j + k) & 1) << 7);
#pragma unroll
    for (int e = 0; e < 2; e++) {
      int x[3];
      const bool in = cell(q, e, x);
      const int c = colour_of(x);
      rs[c * A.P * plane + q] = in ? r0[c * G.half + G.at(x[0] >> 1, x[1], x[2])] : V();
    }
  }
  double res = 0.0, epssq = 0.0, inv_factor2 = 0.0, inv_ncell = 0.0;
  const int itermax = st->s.itermax;
  if (!work) {
    res = st->s.res;
    epssq = st->s.epssq;
    inv_factor2 = st->inv_factor2;
    inv_ncell = st->inv_ncell;
  }
  if (tid == 0) go = 1;
  cluster_barrier(A.blocks);
  const bool low = rank > 0, high = rank < A.blocks - 1;
  unsigned flags = 0u;  // of the thread's first four pairs
  if (work)
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (tid + u * workers < mine) flags |= (unsigned)flag[tid + u * workers] << (8 * u);
  int n = 1;
  V acc{};
  // one colour of an iteration: reads copy `from` (its own cells; the other
  // colour's from `to` once they are new there), writes copy `to`
  const auto half_pass = [&](int from, int to, int h) {
    const V *const own = cells + (2 * from + h) * size + plane;
    const V *const o = cells + (2 * (h ? to : from) + 1 - h) * size + plane;
    V *const out = cells + (2 * to + h) * size + plane;
    const V *const r = rs + h * A.P * plane;
    unsigned fs = flags;
    for (int q = tid, u = 0; q < mine; q += workers, u++) {
      const int f = u < 4 ? (int)(fs & 255u) : flag[q];
      fs >>= 8;
      const bool left = (f >> 7) == h;  // the colour's cell is the pair's left one
      if ((f & 64) && !left) continue;
      // a neighbour beyond a wall is the cell itself: selected addresses, no branches
      const V *const cq = own + q, *const oq = o + q;
      const V c = *cq;
      const V in = *(f & 64 ? cq : oq);
      const V side = *(f & (left ? 1 : 2) ? oq + (left ? -1 : 1) : cq);
      const V s = *(f & 4 ? oq - np : cq), nn = *(f & 8 ? oq + np : cq);
      const V b = *(f & 16 ? oq - plane : cq), t = *(f & 32 ? oq + plane : cq);
      const V D = change<CUBE>(C, c, in, side, s, nn, b, t, r[q]);
      const V m = moved(c, D);
      add_square(acc, D);
      out[q] = m;
      // the planes beside the slab's ends are also the neighbours'
      if (low && q < plane) store_in(in_block(out + A.P * plane + q, rank - 1), m);
      if (high && q >= mine - plane) store_in(in_block(out + q - mine, rank + 1), m);
    }
  };
  // iteration n's d joins p, and r0 is formed from the new one
  const auto fold = [&] {
    V *const d = cells + 2 * (n & 1) * size;
    for (int q = tid; q < mine; q += blockDim.x)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        int x[3];
        if (!cell(q, e, x)) continue;
        const double was = __ldcg(p + (x[2] + 1) * S.g.sk + (x[1] + 1) * S.g.sj + x[0] + 1);
        store_p(G, S.g, p, x[0], x[1], x[2], plus(was, d[colour_of(x) * size + plane + q], unit));
      }
    cluster_barrier(A.blocks);
    for (int q = tid; q < 2 * size; q += blockDim.x) d[q] = V();
    for (int q = tid; q < mine; q += blockDim.x)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        int x[3];
        if (!cell(q, e, x)) continue;
        const int c = (x[2] + 1) * S.g.sk + (x[1] + 1) * S.g.sj + x[0] + 1;
        rs[colour_of(x) * A.P * plane + q] =
            to_cell(-S.factor * residual_of<true>(S, p, rhs, c), V());
      }
    if (rank == 0 && tid == 0) st->base = n;
    cluster_barrier(A.blocks);
  };
  int fold_at = next_fold(n);
  for (;;) {
    if (n == fold_at) {
      fold();
      fold_at = next_fold(n);
    }
    const int from = n & 1, to = from ^ 1;
    if (work) {
      acc = V();
      half_pass(from, to, 0);
    } else if (n > 1) {  // iteration n's squares in this block
      const int w = (tid - workers) >> 5;
      V v[2] = {};
      for (int q = lane + 32 * w; q < workers; q += 64 * kFoldWarps)
#pragma unroll
        for (int u = 0; u < 2; u++)
          if (q + 32 * kFoldWarps * u < workers)
            v[u] = join_u(v[u], scaled(squares[q + 32 * kFoldWarps * u], down));
      const V sum = warp_total_u(join_u(v[0], v[1]));
      if (lane < A.blocks) store_in(in_block(total + rank * kFoldWarps + w, lane), sum);
    }
    cluster_barrier(A.blocks);
    if (work) {
      half_pass(from, to, 1);
      squares[tid] = acc;
    } else if (n > 1) {  // whether it was the last
      V v{};
#pragma unroll
      for (int u = 0; u < 16 * kFoldWarps; u += 32)
        if (lane + u < A.blocks * kFoldWarps) v = join_u(v, total[lane + u]);
      res = (res + as_double(warp_total_u(v)) * inv_factor2) * inv_ncell;
      if (tid == workers && !(res >= epssq && n < itermax)) go = 0;
    }
    cluster_barrier(A.blocks);
    if (!go) break;
    n++;
  }
  // iteration n's d, as the sweeps leave it
  V *const d = n & 1 ? d1 : d0;
  for (int q = tid; q < mine; q += blockDim.x)
#pragma unroll
    for (int e = 0; e < 2; e++) {
      int x[3];
      if (!cell(q, e, x)) continue;
      const int c = colour_of(x);
      d[c * G.half + G.at(x[0] >> 1, x[1], x[2])] = cells[(2 * (n & 1) + c) * size + plane + q];
    }
  if (rank == 0 && tid == (int)blockDim.x - 1) {
    st->s.res = res;
    st->s.it = n;
    st->s.done = 1;
  }
}

constexpr int kFoldMax = 1024;   // block sums that each block of the next sweep folds itself

int up(int a, int b) { return (a + b - 1) / b; }

int sm_count()
{
  int dev = 0, n = 152;
  if (cudaGetDevice(&dev) == cudaSuccess)
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n;
}

// Tile and depth of a sweep. Rows of at most kPairs pairs are whole (no ring
// in x); longer ones are cut evenly. Rows and planes per block: the least time
// of the busiest SM, steps x (0.20 us + 0.035 us for each warp it holds), as
// measured at 64^3, 128^3 and 200 x 40 x 40 over 4-10 rows and 2-32 planes
// (the 0.20 us are the two dependent updates of a step, the rest their issue;
// a launch adds about 3 us whatever the shape).
SweepArgs sweep_shape(int nx, int ny, int nz)
{
  constexpr int kPairs = 64;
  SweepArgs a;
  a.nx = nx;
  a.ny = ny;
  a.nz = nz;
  a.np = up(nx, 2);
  a.pitch = a.np * (ny + 2);
  a.half = a.pitch * (nz + 4);
  const int gx = a.np <= kPairs ? 1 : up(a.np, kPairs - 2);
  a.own = up(a.np, gx);
  a.halo = gx > 1 ? 1 : 0;
  const int pw = a.own + 2 * a.halo, sms = sm_count();
  double best = 1e300;
  a.rows = 1;
  a.kb = nz;
  for (int rows = 1; rows <= 40; rows++) {
    const int threads = up(pw * (rows + 2), 32) * 32;
    if (threads > kMaxThreads) break;
    for (int kb = 1; kb <= nz && kb <= 64; kb++) {
      const int64_t blocks = (int64_t)gx * up(ny, rows) * up(nz, kb);
      const double warps = (double)((blocks + sms - 1) / sms) * (threads / 32);
      const double cost = (kb + 3) * (0.20 + 0.035 * warps);
      if (cost < best) {
        best = cost;
        a.rows = rows;
        a.kb = kb;
      }
    }
  }
  return a;
}

// The slabs of a cluster of `blocks` and its shared memory.
size_t cluster_shape(ClusterArgs &a, const int (&n)[3], int blocks, int threads)
{
  int slab = 2;
  for (int q = 1; q >= 0; q--)
    if (n[q] > n[slab]) slab = q;
  int row = slab == 0 ? 1 : 0, mid = 3 - slab - row;
  if (n[mid] > n[row]) std::swap(row, mid);
  a.axis[0] = row;
  a.axis[1] = mid;
  a.axis[2] = slab;
  for (int q = 0; q < 3; q++) a.n[q] = n[a.axis[q]];
  a.np = up(a.n[0], 2);
  a.plane = a.np * a.n[1];
  a.blocks = blocks;
  a.P = up(a.n[2], blocks);
  const auto magic = [](int d) { return d > 1 ? (unsigned)(((1ull << 32) + d - 1) / d) : 0u; };
  a.mrow = magic(a.np);
  a.mpl = magic(a.plane);
  return 8 * (4 * (size_t)(a.P + 2) * a.plane + 2 * (size_t)a.P * a.plane + threads) +
         (size_t)a.P * a.plane;
}

}  // namespace

// what a solver keeps for its sweeps: the shape, and the device memory (two
// copies of d, and r0; null where the grid is beyond their 32-bit offsets or
// the memory is not to be had: then every iteration runs on p)
struct RbPlan {
  SweepArgs a;
  dim3 grid;
  int threads = 0, blocks = 0;
  size_t smem = 0;
  bool cube = false;  // one spacing on all axes
  void *cells = nullptr;
  // the cluster of a small grid (threads 0: none)
  ClusterArgs c;
  int cluster_threads = 0;
  size_t cluster_smem = 0;
};

namespace {

// programmatic launch: the next sweep's blocks come in while the last of this
// one's leave (and without it each launch took a multiple of 2.05 us)
template <typename V>
bool launch_sweep(const RbPlan &P, const Consts<V> &C, const V *d, V *dout, const V *r0,
    RbState *st, const V *part_in, V *part_out, int n, int np, float down)
{
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = P.grid;
  cfg.blockDim = dim3(P.threads);
  cfg.dynamicSmemBytes = P.smem;
  cfg.stream = stream();
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, P.cube ? k_rb_sweep<V, true> : k_rb_sweep<V, false>, P.a, C, d, dout, r0,
      st, part_in, part_out, n, np, down);
  return launched("k_rb_sweep");
}

template <typename V>
bool cluster_config(const RbPlan &P, cudaLaunchConfig_t &cfg, cudaLaunchAttribute &at)
{
  auto kernel = P.cube ? k_rb_cluster<V, true> : k_rb_cluster<V, false>;
  cfg = {};
  cfg.gridDim = dim3(P.c.blocks);
  cfg.blockDim = dim3(P.cluster_threads);
  cfg.dynamicSmemBytes = P.cluster_smem;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = P.c.blocks;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  // (the same limit from every solver and thread: the attribute is the process's)
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
             (int)kClusterSmem) == cudaSuccess &&
         cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
             cudaSuccess;
}

template <typename V>
bool launch_cluster(const RbPlan &P, const Consts<V> &C, const SorArgs &S, double *p,
    const double *rhs, const V *r0, V *const (&d)[2], double unit, RbState *st, float down)
{
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at;
  if (!cluster_config<V>(P, cfg, at)) return cuda_ok(cudaGetLastError(), "k_rb_cluster attributes");
  cfg.stream = stream();
  const V f[3] = { C.fx, C.fy, C.fz };
  Consts<V> T = C;
  T.fx = f[P.c.axis[0]];
  T.fy = f[P.c.axis[1]];
  T.fz = f[P.c.axis[2]];
  cudaLaunchKernelEx(&cfg, P.cube ? k_rb_cluster<V, true> : k_rb_cluster<V, false>, P.c, P.a, T, S, p,
      rhs, r0, d[0], d[1], unit, st, down);
  return launched("k_rb_cluster");
}

// The cluster for a grid, or none. Pairs: as few blocks as leave each at most a
// pair of cells for each of 256 workers, else sixteen, with 512 workers from
// two pairs each on, up to three (48 thousand cells): an iteration takes 2.3 us
// at 20^3, 2.8 at 30^3, 3.2 at 64 x 10 x 61, 4.8-5.3 at 40^3, sweeps 4.4, 4.3, 4.4
// and 4.9. Doubles: the FP64 pipe of sixteen SMs takes over sooner, 2.9 us at
// 12^3, 3.9 at 20^3 and 7.1 at 30^3 against 5.5, 5.1 and 5.1.
template <typename V>
void choose_cluster(RbPlan &P)
{
  constexpr bool pairs = std::is_same_v<V, df::f2>;
  constexpr int kEach = pairs ? 256 : 64, kMore = pairs ? 512 : 128, kMost = pairs ? 1536 : 450;
  const int n[3] = { P.a.nx, P.a.ny, P.a.nz };
  int threads = 0;
  for (int blocks = 1; blocks <= 16; blocks *= 2) {
    cluster_shape(P.c, n, blocks, 0);
    const int mine = P.c.P * P.c.plane;
    if (mine > kEach && blocks < 16) continue;
    if (mine > kMost) return;
    const int workers = mine > kMore ? 512 : pairs ? 256 : 128;
    threads = workers + 32 * kFoldWarps;
    P.cluster_smem = cluster_shape(P.c, n, blocks, threads);
    break;
  }
  if (P.cluster_smem > kClusterSmem) return;
  P.cluster_threads = threads;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at;
  int fit = 0;
  if (!cluster_config<V>(P, cfg, at) ||
      cudaOccupancyMaxActiveClusters(&fit, P.cube ? k_rb_cluster<V, true> : k_rb_cluster<V, false>,
          &cfg) != cudaSuccess ||
      fit < 1) {
    cudaGetLastError();
    P.cluster_threads = 0;
  }
}

template <typename V>
double sweep_solve(Solver *s, SolverState *ss, const SorArgs &A, double *p, const double *rhs)
{
  const Dims &g = A.g;
  const RbPlan &P = *ss->rb_plan;
  const SweepArgs &a = P.a;
  // (with a factor of zero, or one that has lost bits, the sum of D^2 does not give that of r^2)
  const bool sweeps = P.cells != nullptr && std::isnormal(A.factor);
  const int nb = sweeps ? P.blocks : 0, nb1 = 2 * sor_blocks(A);
  const bool folded = nb > kFoldMax;
  // the first iteration's sums, then the sweeps' two lists and one value for each
  if (!reduce_scratch_alloc(ss->red, nb1 > 2 * nb + 2 ? nb1 : 2 * nb + 2)) return NAN;
  V *const lists = reinterpret_cast<V *>(ss->red.partials);
  V *const part[2] = { lists, lists + nb };
  V *const sum[2] = { lists + 2 * nb, lists + 2 * nb + 1 };
  V *const cells = reinterpret_cast<V *>(P.cells);
  V *const d[2] = { cells, cells + 2 * (size_t)a.half };
  V *const r0 = d[1] + 2 * (size_t)a.half;
  const Consts<V> C = consts(A, V());
  const int scale = sweeps ? -std::ilogb(A.factor) : 0;  // of d and r0
  const double unit = std::ldexp(1.0, -scale);
  SorArgs S = A;
  S.factor = std::ldexp(A.factor, scale);
  // of the sums: 2^-k, with eps^2 2^-k at least 2^-101 (eps below 1 here)
  const int k = std::is_same_v<V, double> || !(s->eps > 0.0)
                    ? 0
                    : std::max(0, std::min(30, 101 + 2 * std::ilogb(s->eps)));
  const float down = std::ldexp(1.0f, -k);
  cudaStream_t q = stream();
  RbState *st = ss->d_rb, *h = ss->h_rb;
  memset(h, 0, sizeof(*h));
  h->s.res = 1.0;
  h->s.epssq = s->eps * s->eps;
  h->s.itermax = s->itermax;
  h->s.ncell = (double)(g.imax * g.jmax * g.kmax);
  h->inv_ncell = 1.0 / h->s.ncell;
  h->inv_factor2 = std::ldexp(1.0 / (S.factor * S.factor), k);
  h->base = s->itermax;  // p holds every iteration until k_rb_open
  h->s.done = !((h->s.res >= h->s.epssq) && (0 < h->s.itermax));
  if (h->s.done) return h->s.res;
  if (!cuda_ok(cudaMemcpyAsync(st, h, sizeof(RbState), cudaMemcpyHostToDevice, q),
          "solve state upload"))
    return NAN;
  // the first iteration runs on p
  const auto on_p = [&](int count) {
    for (int c = 0; c < count; c++)
      if (!launch_rb_iteration(A, p, rhs, &st->s, ss->red, !ss->ext.arith_fp64)) return false;
    return true;
  };
  if (!on_p(1)) return NAN;
  int n = 1;
  const auto open = [&] {
    k_rb_open<V><<<(unsigned)up(a.half, 256), 256, 0, q>>>(a, S, p, rhs, d[n & 1], r0, st, n);
    return launched("k_rb_open");
  };
  const auto close = [&](int at) {
    k_rb_close<V><<<(unsigned)up(a.np * a.ny * a.nz, 256), 256, 0, q>>>(a, g, p, d[0], d[1], unit,
        st, at);
    return launched("k_rb_close");
  };
  const auto fold = [&](int at) {
    k_rb_fold<<<1, 1024, 0, q>>>(st, part[at], nb, sum[at]);
    return launched("k_rb_fold");
  };
  // queue iterations in chunks; the first chunk matches the previous solve's count
  // (how many are queued at once is all that an earlier solve decides)
  int chunk = ss->last_iterations > 0 ? ss->last_iterations - 1 : 16;
  while (!h->s.done) {
    if (!sweeps) {
      const int count = chunk < s->itermax - n ? chunk : s->itermax - n;
      if (!on_p(count)) return NAN;
      n += count;
    } else if (chunk > 0 && n < s->itermax) {
      if (n == 1 && !open()) return NAN;
      if (P.cluster_threads) {  // to the end
        if (!launch_cluster<V>(P, C, S, p, rhs, r0, d, unit, st, down)) return NAN;
        n = s->itermax;
      }
      for (int c = 0; c < chunk && n < s->itermax; c++) {
        n++;
        const int in = (n - 1) & 1, out = n & 1;
        const bool first = n == 2;
        if (folded && !first && !fold(in)) return NAN;
        if (!launch_sweep<V>(P, C, d[in], d[out], r0, st, folded ? sum[in] : part[in], part[out], n,
                first ? 0 : folded ? 1 : nb, down))
          return NAN;
        if (n == next_fold(n - 1) && n < s->itermax && !(close(n) && open())) return NAN;
      }
      if (!P.cluster_threads) {
        // (the sum in the order of the next sweep, which forms the same residual)
        if (folded && !fold(n & 1)) return NAN;
        k_rb_finish<<<1, 32, 0, q>>>(st, folded ? sum[n & 1] : part[n & 1], n, folded ? 1 : nb);
        if (!launched("k_rb_finish")) return NAN;
      }
      if (!close(0)) return NAN;
    }
    if (!cuda_ok(cudaMemcpyAsync(h, st, sizeof(RbState), cudaMemcpyDeviceToHost, q),
            "solve state download"))
      return NAN;
    if (!cuda_ok(cudaStreamSynchronize(q), "solve sync")) return NAN;
    chunk = ss->last_iterations > 64 ? ss->last_iterations / 8 : 8;
  }
  return h->s.res;
}

}  // namespace

// shape and device memory of the sweeps on a grid
bool rb_sweep_alloc(SolverState *ss, const Dims &g, bool cube)
{
  if (ss->rb_plan && ss->rb_plan->a.nx == g.imax && ss->rb_plan->a.ny == g.jmax &&
      ss->rb_plan->a.nz == g.kmax && ss->rb_plan->cube == cube)
    return true;
  rb_sweep_free(ss);
  RbPlan *P = ss->rb_plan = new RbPlan();
  SweepArgs &a = P->a = sweep_shape(g.imax, g.jmax, g.kmax);
  const int pw = a.own + 2 * a.halo;
  P->threads = up(pw * (a.rows + 2), 32) * 32;
  P->grid = dim3(up(a.np, a.own), up(a.ny, a.rows), up(a.nz, a.kb));
  P->blocks = (int)(P->grid.x * P->grid.y * P->grid.z);
  P->cube = cube;
  P->smem = 2 * (size_t)pw * (a.rows + 2 + a.rows + 4) * 8;
  const int64_t half = (int64_t)a.np * (a.ny + 2) * (a.nz + 4);
  if (2 * half < ((int64_t)1 << 31) &&
      cudaMalloc(&P->cells, 3 * 2 * (size_t)half * 8) != cudaSuccess) {
    cudaGetLastError();
    P->cells = nullptr;
  }
  if (P->cells && ss->ext.arith_fp64) choose_cluster<double>(*P);
  if (P->cells && !ss->ext.arith_fp64) choose_cluster<df::f2>(*P);
  return cuda_ok(cudaMalloc(&ss->d_rb, sizeof(RbState)), "cudaMalloc(rb state)") &&
         cuda_ok(cudaMallocHost(&ss->h_rb, sizeof(RbState)), "cudaMallocHost(rb state)");
}

void rb_sweep_free(SolverState *ss)
{
  if (ss->d_rb) cudaFree(ss->d_rb);
  if (ss->h_rb) cudaFreeHost(ss->h_rb);
  ss->d_rb = ss->h_rb = nullptr;
  if (!ss->rb_plan) return;
  if (ss->rb_plan->cells) cudaFree(ss->rb_plan->cells);
  delete ss->rb_plan;
  ss->rb_plan = nullptr;
}

double rb_sweep_solve(Solver *s, SolverState *ss, const SorArgs &A, double *p, const double *rhs)
{
  return ss->ext.arith_fp64 ? sweep_solve<double>(s, ss, A, p, rhs)
                            : sweep_solve<df::f2>(s, ss, A, p, rhs);
}

}  // namespace nusif
