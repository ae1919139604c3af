// Kernel templates for the nLPT field pipeline: FFT passes with fused
// prologues/epilogues.  Data layout (same as Grid_FFT<real_t>, grid_fft.cc:45):
//   real space   [n0][n1][n2+2] reals, row-major (grid_fft.hh:184-188)
//   k space      [n0][n1][n2/2+1] complex, in place (grid_fft.hh:196-200)
// with i <-> kx, j <-> ky, k <-> kz >= 0 on a single device.
//
// Passes:
//   strided pass  (axis 0 or 1): one CTA owns NCOL consecutive kz columns of
//                 one slab; element e of column c lives at smem[e*NCOL + c],
//                 threads are column-fastest so every global row access is a
//                 contiguous NCOL*sizeof(complex) segment.
//   z pass        (axis 2): one thread group per line, lines contiguous in
//                 HBM; real transforms use the half-length complex packing.
#pragma once

#include <type_traits>

#include "mf_fft.cuh"
#include "mf_fx.cuh"
#include "mf_tma.cuh"

// largest radix of the pipelined strided passes' plans (a build-time knob)
#ifndef MF_COL_MAXR
#define MF_COL_MAXR 8
#endif

namespace mf {

// minimum resident CTAs per SM a pipelined strided pass is compiled for (its
// __launch_bounds__): threads per CTA, values per thread E of the plan, bytes
// per scalar.  Sized from the registers the plan needs (~4 per scalar held,
// plus 32), at most 4: without the bound the 128-thread FP32 CTAs took up to
// 255 registers (8 warps per SM).
__host__ __device__ constexpr int col_minb(int threads, int e, int scalar_bytes) {
  int need = 4 * e * (scalar_bytes / 4) + 32;
  if (scalar_bytes == 8 && need > 168) need = 168;  // fixed-point FP64 columns: three 128-thread CTAs
  need = need < 64 ? 64 : (need > 255 ? 255 : need);
  const int b = 65536 / (threads * need);
  return b < 1 ? 1 : (b > 4 ? 4 : b);
}

// exchange layout of a pipelined strided tile [row e][NCOL columns]: the
// row swizzle (pidx<2>) where a row is 64 bytes (8 FP32 or 4 FP64 complex
// columns) and the op asks for it (kColSwizzle), identity otherwise.  The
// swizzle's per-element address arithmetic costs registers: the ops with a
// prologue or a prefetched read-modify-write target (x passes) sit at the
// 128-register cap of two CTAs per SM and would spill, so they keep the
// identity layout.
template <class OP, class = void>
struct col_swizzle : std::false_type {};
template <class OP>
struct col_swizzle<OP, std::void_t<decltype(OP::kColSwizzle)>> : std::integral_constant<bool, OP::kColSwizzle> {};
template <typename T, int NCOL, class OP>
__host__ __device__ constexpr int col_layout() {
  return (col_swizzle<OP>::value && NCOL * (int)sizeof(cplx<T>) == 64) ? 2 : 0;
}

// the plain N-grid passes
template <class OP>
struct plain_op : std::false_type {};
template <typename T, int L, int AXIS>
struct plain_op<PlainStridedOp<T, L, AXIS>> : std::true_type {};

// whether a pass transforms its lines in fixed point: FP64, unless the op asks
// for FP64 butterflies
template <class OP, class = void>
struct butterfly_op : std::false_type {};
template <class OP>
struct butterfly_op<OP, std::void_t<decltype(OP::kButterflies)>> : std::true_type {};
template <typename T, class OP>
__host__ __device__ constexpr bool fixed_point_lines() {
  return sizeof(T) == 8 && !butterfly_op<OP>::value;
}

// ops with a per-tile prologue (tile_prep / xform_tile) in the pipelined pass
template <class OP, class = void>
struct has_tile_prep : std::false_type {};
template <class OP>
struct has_tile_prep<OP, std::void_t<decltype(&OP::tile_prep)>> : std::true_type {};

// ---------------------------------------------------------------------------
// strided pass producing three transforms per column (three-component
// assembly): the loader yields the three inputs of each element at once.
// FP32: the first component stays in
// registers, the other two go to their own tiles as they are loaded, and each
// later component's transform runs from (and exchanges through) its tile, so
// registers hold one component and two CTAs share an SM (one's loads overlap
// the other's transforms).  Every thread reads back only the tile slots it
// wrote (the first stage's inputs), so no barrier precedes the reads.
template <typename T, int L, bool INV, int NCOL, class OP, int MINB>
__global__ void __launch_bounds__(NCOL * LineFFT<T, L, INV>::TPL, MINB)
k_colfft3s(OP op, const cplx<T>* __restrict__ tw, int ncols) {
  using F = LineFFT<T, L, INV>;
  using C = cplx<T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* xchg = reinterpret_cast<C*>(smem_raw);  // exchanges of the first component
  C* tile1 = xchg + L * NCOL;
  C* tile2 = tile1 + L * NCOL;
  const int c = threadIdx.x, t = threadIdx.y;
  const int col = blockIdx.x * NCOL + c;
  const int slab = blockIdx.y;
  const bool valid = col < ncols;
  if constexpr (sizeof(T) == 8) {
#pragma unroll 1
    for (int i = 0; i < F::E; ++i) {
      C w[3] = {mkc<T>(T(0), T(0)), mkc<T>(T(0), T(0)), mkc<T>(T(0), T(0))};
      if (valid) op.load3(slab, t + i * F::TPL, col, w);
      const int o = tile_slot<F, NCOL>(t, i) + c;
      xchg[o] = w[0];
      tile1[o] = w[1];
      tile2[o] = w[2];
    }
#pragma unroll 1
    for (int d = 0; d < 3; ++d) {
      C* tl = xchg + d * L * NCOL;
      const int xs = col_fx<F, NCOL>(tl, t, c, tw);
      if (valid) {
#pragma unroll 2
        for (int i = 0; i < F::E; ++i)
          op.store(d, slab, t + i * F::TPL, col,
                   fx::to_c(reinterpret_cast<const longlong2*>(tl)[tile_slot<F, NCOL>(t, i) + c], xs));
      }
    }
    return;
  }
  C v[F::E];
#pragma unroll
  for (int s = 0; s < F::E; ++s) {
    const int e = F::in_index(t, s);
    C w[3] = {mkc<T>(T(0), T(0)), mkc<T>(T(0), T(0)), mkc<T>(T(0), T(0))};
    if (valid) op.load3(slab, e, col, w);
    v[s] = w[0];
    tile1[e * NCOL + c] = w[1];
    tile2[e * NCOL + c] = w[2];
  }
  F::run(v, t, xchg + c, NCOL, tw, SyncBlock{});
  if (valid) {
#pragma unroll
    for (int s = 0; s < F::E; ++s) op.store(0, slab, F::out_index(t, s), col, v[s]);
  }
#pragma unroll
  for (int d = 1; d < 3; ++d) {
    C* tl = (d == 1) ? tile1 : tile2;
#pragma unroll
    for (int s = 0; s < F::E; ++s) v[s] = tl[F::in_index(t, s) * NCOL + c];
    F::run(v, t, tl + c, NCOL, tw, SyncBlock{});
    if (valid) {
#pragma unroll
      for (int s = 0; s < F::E; ++s) op.store(d, slab, F::out_index(t, s), col, v[s]);
    }
  }
}

// ---------------------------------------------------------------------------
// persistent strided pass of the FP64 lines and of the FP32 lengths without a
// two-stage plan (k_col2 below; double-buffered in FP32).  Each CTA walks tiles
// (column tile, slab, operand) with stride gridDim.x; while a tile is being
// transformed, the raw elements of the CTA's next tile are already being
// copied into the other shared-memory buffer with cp.async.  Every thread
// copies exactly the elements it reads for its first FFT stage, so a
// per-thread wait_group suffices before the read.
// OP: src_ok(e) (else the element is zero), gap(e) (zero for every thread,
//     known at compile time), srcp(z, slab, e, col) -> const C*,
//     xform(z, slab, e, col, raw), store_z(z, slab, e, col, v)
//     (+ kPrefetch: prefetch/store_pre on the same coordinates)
// ---------------------------------------------------------------------------
// the tile a persistent CTA works on, (column tile, slab, operand), stepped by
// the grid size with carries instead of a division per tile
struct TilePos {
  int ct, slab, z;
  __device__ __forceinline__ static TilePos of(int tl, int ntc, int nslab) {
    TilePos p;
    p.ct = tl % ntc;
    const int r = tl / ntc;
    p.slab = r % nslab;
    p.z = r / nslab;
    return p;
  }
  // step: the position of tile index gridDim.x
  __device__ __forceinline__ TilePos next(const TilePos& step, int ntc, int nslab) const {
    TilePos p{ct + step.ct, slab + step.slab, z + step.z};
    if (p.ct >= ntc) { p.ct -= ntc; ++p.slab; }
    if (p.slab >= nslab) { p.slab -= nslab; ++p.z; }
    return p;
  }
};

template <typename T, int L, bool INV, int NCOL, class OP>
__global__ void __launch_bounds__(NCOL * LineFFT<T, L, INV, MF_COL_MAXR>::TPL,
                                  col_minb(NCOL * LineFFT<T, L, INV, MF_COL_MAXR>::TPL,
                                           LineFFT<T, L, INV, MF_COL_MAXR>::E, (int)sizeof(T)))
k_colfft_pipe(OP op, const cplx<T>* __restrict__ tw, int ncols, int ntc, int nslab, int nz) {
  constexpr int LAY = col_layout<T, NCOL, OP>();
  using F = LineFFT<T, L, INV, MF_COL_MAXR, LAY>;
  using C = cplx<T>;
  using I = LineIdx<F::TPL>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf0 = reinterpret_cast<C*>(smem_raw);
  [[maybe_unused]] C* buf1 = buf0 + L * NCOL;
  const int c = threadIdx.x, t = threadIdx.y;
  const int total = ntc * nslab * nz;
  auto issue = [&](const TilePos& p, C* buf) {
    const int col = p.ct * NCOL + c;
#pragma unroll
    for (int s = 0; s < F::E; ++s) {
      C* d = buf + F::in_slot(t, s) * NCOL + c;
      const I e{t, F::in_const(s)};
      if (col < ncols && op.src_ok(e)) {
        const C* g = op.srcp(p.z, p.slab, e, col);
        if constexpr (sizeof(C) == 16) cp_async16(d, g); else cp_async8(d, g);
      } else {
        *d = mkc<T>(T(0), T(0));
      }
    }
    cp_async_commit();
  };
  if constexpr (fixed_point_lines<T, OP>()) {
    // FP64 columns in fixed point: bound by the integer pipes, so one buffer
    // per CTA and more CTAs per SM instead of a second buffer
    const TilePos step = TilePos::of(gridDim.x, ntc, nslab);
    TilePos p = TilePos::of(blockIdx.x, ntc, nslab);
    for (int tl = blockIdx.x; tl < total; tl += gridDim.x, p = p.next(step, ntc, nslab)) {
      issue(p, buf0);
      cp_async_wait<0>();
      const int col = p.ct * NCOL + c;
      if constexpr (has_tile_prep<OP>::value) {
        const auto tp = op.tile_prep(p.z, p.slab, col);
#pragma unroll 2
        for (int i = 0; i < F::E; ++i) {
          const int o = tile_slot<F, NCOL>(t, i) + c;
          if (op.src_ok(t + i * F::TPL)) buf0[o] = op.xform_tile(tp, t + i * F::TPL, buf0[o]);
        }
      }
      const int xs = col_fx<F, NCOL>(buf0, t, c, tw);
      if (col < ncols) {
#pragma unroll 2
        for (int i = 0; i < F::E; ++i)
          op.store_z(p.z, p.slab, t + i * F::TPL, col,
                     fx::to_c(reinterpret_cast<const longlong2*>(buf0)[tile_slot<F, NCOL>(t, i) + c], xs));
      }
      // (a thread's next copies overwrite only elements that it read itself)
    }
    return;
  }
  int tl = blockIdx.x;
  const TilePos step = TilePos::of(gridDim.x, ntc, nslab);
  TilePos nx = TilePos::of(tl, ntc, nslab);
  if (tl < total) issue(nx, buf0); else cp_async_commit();
  for (int it = 0; tl < total; tl += gridDim.x, ++it) {
    C* cur = (it & 1) ? buf1 : buf0;
    C* nxt = (it & 1) ? buf0 : buf1;
    const TilePos p = nx;
    nx = p.next(step, ntc, nslab);
    if (tl + (int)gridDim.x < total) issue(nx, nxt); else cp_async_commit();
    cp_async_wait<1>();
    const int col = p.ct * NCOL + c;
    const bool valid = col < ncols;
    C v[F::E];
    if constexpr (has_tile_prep<OP>::value) {
      const auto tp = op.tile_prep(p.z, p.slab, col);
#pragma unroll
      for (int s = 0; s < F::E; ++s)
        v[s] = op.xform_tile(tp, I{t, F::in_const(s)}, cur[F::in_slot(t, s) * NCOL + c]);
    } else {
#pragma unroll
      for (int s = 0; s < F::E; ++s)
        v[s] = op.xform(p.z, p.slab, I{t, F::in_const(s)}, col, cur[F::in_slot(t, s) * NCOL + c]);
    }
    if constexpr (OP::kPrefetch) {
      C pre[F::E];
#pragma unroll
      for (int s = 0; s < F::E; ++s)
        pre[s] = valid ? op.prefetch(p.slab, I{t, F::out_const(s)}, col) : mkc<T>(T(0), T(0));
      F::run(v, t, cur + c, NCOL, tw, SyncBlock{});
      if (valid) {
#pragma unroll
        for (int s = 0; s < F::E; ++s) op.store_pre(p.slab, I{t, F::out_const(s)}, col, v[s], pre[s]);
      }
    } else {
      F::run(v, t, cur + c, NCOL, tw, SyncBlock{});
      if (valid) {
#pragma unroll
        for (int s = 0; s < F::E; ++s) op.store_z(p.z, p.slab, I{t, F::out_const(s)}, col, v[s]);
      }
    }
    __syncthreads();  // cur is refilled by the next iteration's copies
  }
  cp_async_wait<0>();
}

// ---------------------------------------------------------------------------
// Two-stage strided pass (FP32): a column of length L = R1 R2 as one radix-R1
// and one radix-R2 butterfly with a single exchange between them, where the
// radix-8 plans take three stages and two exchanges.  At those plans the
// passes spent ~70% of the shared-memory pipe and half of the issue slots;
// a stage less takes a quarter of the shared-memory accesses, three of the five
// CTA barriers per tile and one set of twiddles away.
//   stage 1: butterfly b in [0, R2) takes rows b + p R2, leaves q at row b R1 + q
//   stage 2: butterfly k in [0, R1) takes rows k + p R1 (times w_L^(pk)),
//            outputs row k + q R1
// Threads are column-fastest, (b or k) = threadIdx.y; the stages use R2 and R1
// of them (whole warps idle in the smaller one).  In the exchange the low row
// bit is flipped by the parity of b, so that the two rows of a half-warp fall
// on different banks.
// ---------------------------------------------------------------------------
// (measured per launch, before -> after: y c2r of an operand pair 22.1 -> 17.2
// us at L = 192, 70.0 -> 52.1 at 288, 142 -> 121 at 384, of three operands 1176
// -> 979 us at 768; N-grid passes 292 -> 229 us at 512; five aliased
// products at N=256 1430 -> 1309 us with tiles of 16 columns.)
__host__ __device__ constexpr int col2_r1(int L) {
  switch (L) {
    case 128: return 8;
    case 144: return 12;
    case 192: return 12;
    case 256: return 16;
    case 288: return 12;
    case 384: return 16;
    case 512: return 16;
    case 576: return 24;
    case 768: return 24;
    default: return 0;
  }
}
template <int L>
struct Col2 {
  static constexpr int R1 = col2_r1(L), R2 = R1 ? L / R1 : 0;
  static constexpr int TY = R1 > R2 ? R1 : R2;  // threads per column
  static constexpr int RMAX = TY;
};
// resident CTAs per SM, from the registers that the larger butterfly needs
__host__ __device__ constexpr int col2_minb(int threads, int rmax) {
  const int need = rmax >= 32 ? 128 : (rmax >= 24 ? 104 : 80);
  const int b = 65536 / (threads * need);
  return b < 1 ? 1 : b;
}
template <int R1>
__device__ __forceinline__ int col2_out(int b, int q) {  // row of output q of stage-1 butterfly b
  const int f = b & 1;
  return b * R1 + ((q & 1) ? q - f : q + f);
}
template <int R1>
__device__ __forceinline__ int col2_in(int k, int p) {  // row of input p of stage-2 butterfly k
  return p * R1 + ((p & 1) ? (k ^ 1) : k);
}

template <typename T, int L, bool INV, int NCOL, class OP>
__global__ void __launch_bounds__(NCOL * Col2<L>::TY, col2_minb(NCOL * Col2<L>::TY, Col2<L>::RMAX))
k_col2(OP op, const cplx<T>* __restrict__ tw, int ncols, int ntc, int nslab, int nz) {
  constexpr int R1 = Col2<L>::R1, R2 = Col2<L>::R2;
  using C = cplx<T>;
  using I1 = LineIdx<R2>;
  using I2 = LineIdx<R1>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf0 = reinterpret_cast<C*>(smem_raw);
  C* buf1 = buf0 + L * NCOL;
  const int c = threadIdx.x, u = threadIdx.y;
  const int total = ntc * nslab * nz;
  auto issue = [&](const TilePos& p, C* buf) {
    const int col = p.ct * NCOL + c;
    if (R2 == Col2<L>::TY || u < R2) {
#pragma unroll
      for (int s = 0; s < R1; ++s) {
        const I1 e{u, s * R2};
        if (op.gap(e)) continue;  // neither staged nor read
        C* d = buf + (u + s * R2) * NCOL + c;
        if (col < ncols && op.src_ok(e)) cp_async8(d, op.srcp(p.z, p.slab, e, col));
        else *d = mkc<T>(T(0), T(0));
      }
    }
    cp_async_commit();
  };
  int tl = blockIdx.x;
  const TilePos step = TilePos::of(gridDim.x, ntc, nslab);
  TilePos nx = TilePos::of(tl, ntc, nslab);
  if (tl < total) issue(nx, buf0);
  for (int it = 0; tl < total; tl += gridDim.x, ++it) {
    C* cur = (it & 1) ? buf1 : buf0;
    C* nxt = (it & 1) ? buf0 : buf1;
    const TilePos p = nx;
    nx = p.next(step, ntc, nslab);
    if (tl + (int)gridDim.x < total) issue(nx, nxt); else cp_async_commit();
    cp_async_wait<1>();
    const int col = p.ct * NCOL + c;
    const bool act1 = R2 == Col2<L>::TY || u < R2, act2 = (R1 == Col2<L>::TY || u < R1) && col < ncols;
    C v[R1];
    if (act1) {
      if constexpr (has_tile_prep<OP>::value) {
        const auto tp = op.tile_prep(p.z, p.slab, col);
#pragma unroll
        for (int s = 0; s < R1; ++s)
          v[s] = op.gap(I1{u, s * R2}) ? mkc<T>(T(0), T(0))
                                       : op.xform_tile(tp, I1{u, s * R2}, cur[(u + s * R2) * NCOL + c]);
      } else {
#pragma unroll
        for (int s = 0; s < R1; ++s)
          v[s] = op.gap(I1{u, s * R2}) ? mkc<T>(T(0), T(0))
                                       : op.xform(p.z, p.slab, I1{u, s * R2}, col, cur[(u + s * R2) * NCOL + c]);
      }
      dftR<T, INV, R1>(v);
    }
    __syncthreads();  // every input of the tile has been read
    if (act1) {
#pragma unroll
      for (int q = 0; q < R1; ++q) cur[col2_out<R1>(u, q) * NCOL + c] = v[q];
    }
    __syncthreads();
    if (act2) {
      C w[R2];
#pragma unroll
      for (int s = 0; s < R2; ++s) w[s] = cur[col2_in<R1>(u, s) * NCOL + c];
#pragma unroll
      for (int s = 1; s < R2; ++s) w[s] = INV ? cmulc(w[s], tw[s * u]) : cmul(w[s], tw[s * u]);
      dftR<T, INV, R2>(w);
      if constexpr (OP::kPrefetch) {  // a read-modify-write target, eight values in flight
#pragma unroll
        for (int h = 0; h < R2; h += 8) {
          C pre[8];
#pragma unroll
          for (int q = 0; q < 8; ++q)
            if (h + q < R2) pre[q] = op.prefetch(p.slab, I2{u, (h + q) * R1}, col);
#pragma unroll
          for (int q = 0; q < 8; ++q)
            if (h + q < R2) op.store_pre(p.slab, I2{u, (h + q) * R1}, col, w[h + q], pre[q]);
        }
      } else {
#pragma unroll
        for (int q = 0; q < R2; ++q) op.store_z(p.z, p.slab, I2{u, q * R1}, col, w[q]);
      }
    }
    __syncthreads();  // cur is refilled by the next iteration's copies
  }
}

// convolve3's truncation (ConvXTruncOp) in the two-stage form: the forward
// transform's outputs of a thread, rows k + q R1, are the inputs of the
// radix-R2 butterfly that starts the inverse transform (R2, then R1), so the
// truncation and the turn happen in registers: two exchanges in all
template <typename T, int L, int NCOL, class OP>
__global__ void __launch_bounds__(NCOL * Col2<L>::TY, col2_minb(NCOL * Col2<L>::TY, Col2<L>::RMAX))
k_col2_trunc(OP op, const cplx<T>* __restrict__ tw, int ncols, int ntc, int nslab) {
  constexpr int R1 = Col2<L>::R1, R2 = Col2<L>::R2, TY = Col2<L>::TY;
  using C = cplx<T>;
  using I1 = LineIdx<R2>;
  using I2 = LineIdx<R1>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf0 = reinterpret_cast<C*>(smem_raw);
  C* buf1 = buf0 + L * NCOL;
  const int c = threadIdx.x, u = threadIdx.y;
  const int total = ntc * nslab;
  auto issue = [&](const TilePos& p, C* buf) {
    const int col = p.ct * NCOL + c;
    if (R2 == TY || u < R2) {
#pragma unroll
      for (int s = 0; s < R1; ++s) {
        C* d = buf + (u + s * R2) * NCOL + c;
        if (col < ncols) cp_async8(d, op.at(p.slab, I1{u, s * R2}, col));
        else *d = mkc<T>(T(0), T(0));
      }
    }
    cp_async_commit();
  };
  int tl = blockIdx.x;
  const TilePos step = TilePos::of(gridDim.x, ntc, nslab);
  TilePos nx = TilePos::of(tl, ntc, nslab);
  if (tl < total) issue(nx, buf0);
  for (int it = 0; tl < total; tl += gridDim.x, ++it) {
    C* cur = (it & 1) ? buf1 : buf0;
    C* nxt = (it & 1) ? buf0 : buf1;
    const TilePos p = nx;
    nx = p.next(step, ntc, nslab);
    cp_async_wait<0>();
    const int col = p.ct * NCOL + c;
    const bool act1 = R2 == TY || u < R2, act2 = R1 == TY || u < R1;
    {
      C v[R1];
      if (act1) {
#pragma unroll
        for (int s = 0; s < R1; ++s) v[s] = cur[(u + s * R2) * NCOL + c];
        dftR<T, false, R1>(v);
      }
      __syncthreads();  // (as in k_col2)
      if (tl + (int)gridDim.x < total) issue(nx, nxt);
      if (act1) {
#pragma unroll
        for (int q = 0; q < R1; ++q) cur[col2_out<R1>(u, q) * NCOL + c] = v[q];
      }
    }
    __syncthreads();
    C v[R2];
    if (act2) {
#pragma unroll
      for (int s = 0; s < R2; ++s) v[s] = cur[col2_in<R1>(u, s) * NCOL + c];
#pragma unroll
      for (int s = 1; s < R2; ++s) v[s] = cmul(v[s], tw[s * u]);
      dftR<T, false, R2>(v);
#pragma unroll
      for (int q = 0; q < R2; ++q) v[q] = op.mask(p.slab, I2{u, q * R1}, col, v[q]);
      dftR<T, true, R2>(v);
    }
    __syncthreads();  // every input of the second stage has been read
    if (act2) {
#pragma unroll
      for (int q = 0; q < R2; ++q) cur[col2_out<R2>(u, q) * NCOL + c] = v[q];
    }
    __syncthreads();
    if (act1 && col < ncols) {
      C w[R1];
#pragma unroll
      for (int s = 0; s < R1; ++s) w[s] = cur[col2_in<R2>(u, s) * NCOL + c];
#pragma unroll
      for (int s = 1; s < R1; ++s) w[s] = cmulc(w[s], tw[s * u]);
      dftR<T, true, R1>(w);
#pragma unroll
      for (int q = 0; q < R1; ++q) *op.at(p.slab, I1{u, q * R2}, col) = w[q];
    }
  }
}

// ---------------------------------------------------------------------------
// strided forward transform, truncation and inverse transform of one column in
// one pass (ConvXTruncOp), for the lengths that k_colfft_pipe takes and as there
// ---------------------------------------------------------------------------
template <typename T, int L, int NCOL, class OP>
__global__ void __launch_bounds__(NCOL * LineFFT<T, L, false, MF_COL_MAXR>::TPL,
                                  col_minb(NCOL * LineFFT<T, L, false, MF_COL_MAXR>::TPL,
                                           LineFFT<T, L, false, MF_COL_MAXR>::E, (int)sizeof(T)))
k_colfft_trunc(OP op, const cplx<T>* __restrict__ tw, int ncols, int ntc, int nslab) {
  constexpr int LAY = col_layout<T, NCOL, OP>();
  using FF = LineFFT<T, L, false, MF_COL_MAXR, LAY>;
  using FI = LineFFT<T, L, true, MF_COL_MAXR, LAY>;
  static_assert(FF::E == FI::E && FF::TPL == FI::TPL, "one plan for both directions");
  using C = cplx<T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf0 = reinterpret_cast<C*>(smem_raw);
  [[maybe_unused]] C* buf1 = buf0 + L * NCOL;
  const int c = threadIdx.x, t = threadIdx.y;
  using I = LineIdx<FF::TPL>;
  const int total = ntc * nslab;
  auto issue = [&](const TilePos& p, C* buf) {
    const int col = p.ct * NCOL + c;
#pragma unroll
    for (int s = 0; s < FF::E; ++s) {
      C* d = buf + FF::in_slot(t, s) * NCOL + c;
      const C* g = op.at(p.slab, I{t, FF::in_const(s)}, col);
      if (col < ncols) {
        if constexpr (sizeof(C) == 16) cp_async16(d, g); else cp_async8(d, g);
      } else {
        *d = mkc<T>(T(0), T(0));
      }
    }
    cp_async_commit();
  };
  if constexpr (sizeof(T) == 8) {  // one buffer, as in k_colfft_pipe
    const TilePos step = TilePos::of(gridDim.x, ntc, nslab);
    TilePos p = TilePos::of(blockIdx.x, ntc, nslab);
    for (int tl = blockIdx.x; tl < total; tl += gridDim.x, p = p.next(step, ntc, nslab)) {
      issue(p, buf0);
      cp_async_wait<0>();
      const int col = p.ct * NCOL + c;
      int xs = col_fx<FF, NCOL>(buf0, t, c, tw);
#pragma unroll 2
      for (int i = 0; i < FF::E; ++i) {
        const int o = tile_slot<FF, NCOL>(t, i) + c;
        buf0[o] = op.mask(p.slab, t + i * FF::TPL, col, fx::to_c(reinterpret_cast<const longlong2*>(buf0)[o], xs));
      }
      xs = col_fx<FI, NCOL>(buf0, t, c, tw);
      if (col < ncols) {
#pragma unroll 2
        for (int i = 0; i < FF::E; ++i)
          *op.at(p.slab, t + i * FF::TPL, col) =
              fx::to_c(reinterpret_cast<const longlong2*>(buf0)[tile_slot<FF, NCOL>(t, i) + c], xs);
      }
    }
    return;
  }
  int tl = blockIdx.x;
  const TilePos step = TilePos::of(gridDim.x, ntc, nslab);
  TilePos nx = TilePos::of(tl, ntc, nslab);
  if (tl < total) issue(nx, buf0); else cp_async_commit();
  for (int it = 0; tl < total; tl += gridDim.x, ++it) {
    C* cur = (it & 1) ? buf1 : buf0;
    C* nxt = (it & 1) ? buf0 : buf1;
    const TilePos p = nx;
    nx = p.next(step, ntc, nslab);
    if (tl + (int)gridDim.x < total) issue(nx, nxt); else cp_async_commit();
    cp_async_wait<1>();
    const int col = p.ct * NCOL + c;
    const bool valid = col < ncols;
    C v[FF::E];
#pragma unroll
    for (int s = 0; s < FF::E; ++s) v[s] = cur[FF::in_slot(t, s) * NCOL + c];
    FF::run(v, t, cur + c, NCOL, tw, SyncBlock{});
    __syncthreads();  // the last exchange of the forward transform has been read
#pragma unroll
    for (int s = 0; s < FF::E; ++s)
      cur[FF::out_slot(t, s) * NCOL + c] = op.mask(p.slab, I{t, FF::out_const(s)}, col, v[s]);
    __syncthreads();
#pragma unroll
    for (int s = 0; s < FI::E; ++s) v[s] = cur[FI::in_slot(t, s) * NCOL + c];
    FI::run(v, t, cur + c, NCOL, tw, SyncBlock{});
    if (valid) {
#pragma unroll
      for (int s = 0; s < FI::E; ++s) *op.at(p.slab, I{t, FI::out_const(s)}, col) = v[s];
    }
    __syncthreads();  // cur is refilled by the next iteration's copies
  }
  cp_async_wait<0>();
}

// ---------------------------------------------------------------------------
// z pass, real -> half complex (forward), one line per thread group
// OP: __device__ C load_pair(int line, int m) const;   // (x[2m], x[2m+1])
//     __device__ void store(int line, int k, C v) const;  // k in [0, kout)
// ---------------------------------------------------------------------------
// distance between the lines' areas of the plain z passes: the exchange stride
// of the XOR layouts, at least the H+1 values of a half-complex line
template <int H>
__host__ __device__ constexpr int zplain_stride() {
  return zline_stride(H) > H + 1 ? zline_stride(H) : H + 1;
}
template <typename T, int H, int NT, class OP>
__global__ void __launch_bounds__(NT) k_zr2c(OP op, const cplx<T>* __restrict__ twH,
                                               const cplx<T>* __restrict__ twM, int nlines, int kout) {
  constexpr int LAY = zlayout(H);
  using F = LineFFT<T, H, false, 8, LAY>;
  using C = cplx<T>;
  // a line's shared-memory area is its own: warp barriers when its threads sit inside one warp
  using SYNC = typename std::conditional<(F::TPL <= 32 && 32 % F::TPL == 0 && NT % 32 == 0), SyncWarp, SyncBlock>::type;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int t = threadIdx.x, ly = threadIdx.y;
  const int line = blockIdx.x * blockDim.y + ly;
  const bool valid = line < nlines;
  C* sm = reinterpret_cast<C*>(smem_raw) + ly * zplain_stride<H>();
  if constexpr (fixed_point_lines<T, OP>()) {
#pragma unroll 4
    for (int i = 0; i < F::E; ++i)
      sm[t + i * F::TPL] = valid ? op.load_pair(line, t + i * F::TPL) : mkc<T>(T(0), T(0));
    const int xs = r2c_line_to_fx<H, F::TPL, 0>(sm, t, ly, SYNC{});
    longlong2* sx = reinterpret_cast<longlong2*>(sm);
    r2c_line_fx<F, H, 0>(sx, sx, t, twH, SYNC{});
    if (valid) {
#pragma unroll 2
      for (int k = t; k < kout; k += F::TPL) op.store(line, k, r2c_line_out<H, LAY>(sx, k, xs, twM));
    }
    return;
  }
  C v[F::E];
#pragma unroll
  for (int s = 0; s < F::E; ++s) v[s] = valid ? op.load_pair(line, F::in_index(t, s)) : mkc<T>(T(0), T(0));
  F::run(v, t, sm, 1, twH, SYNC{});
  SYNC{}();
#pragma unroll
  for (int s = 0; s < F::E; ++s) sm[F::out_slot(t, s)] = v[s];
  SYNC{}();
  if (valid) {
    for (int k = t; k < kout; k += F::TPL) {
      const C zk = sm[pidx<LAY>(k == H ? 0 : k)];
      const C zc = cconj(sm[pidx<LAY>(k == 0 || k == H ? 0 : H - k)]);
      const C E = mkc<T>(T(0.5) * (zk.x + zc.x), T(0.5) * (zk.y + zc.y));
      // O = (zk - zc) / (2i)
      const C O = mkc<T>(T(0.5) * (zk.y - zc.y), -T(0.5) * (zk.x - zc.x));
      op.store(line, k, cadd(E, cmul(twM[k], O)));
    }
  }
}

// ---------------------------------------------------------------------------
// z pass, half complex -> real (inverse), Re-semantics of FFTW's c2r
// OP: __device__ C load(int line, int k) const;          // k in [0, H]
//     __device__ void store_pair(int line, int m, C v) const;
// ---------------------------------------------------------------------------
template <typename T, int H>
__device__ __forceinline__ cplx<T> c2r_pre(const cplx<T>* sm, int k, const cplx<T>* __restrict__ twM) {
  using C = cplx<T>;
  C A = sm[k];
  C B = cconj(sm[H - k]);
  if (k == 0) { A.y = T(0); B.y = T(0); }
  const C Ev = cadd(A, B);
  const C Ov = cmulc(csub(A, B), twM[k]);  // (A-B) e^{+2 pi i k/M}
  return mkc<T>(Ev.x - Ov.y, Ev.y + Ov.x);  // E + i O
}

template <typename T, int H, int NT, class OP>
__global__ void __launch_bounds__(NT) k_zc2r(OP op, const cplx<T>* __restrict__ twH,
                                               const cplx<T>* __restrict__ twM, int nlines, int kin) {
  using F = LineFFT<T, H, true, 8, zlayout(H)>;
  using C = cplx<T>;
  // a line's shared-memory area is its own: warp barriers when its threads sit inside one warp
  using SYNC = typename std::conditional<(F::TPL <= 32 && 32 % F::TPL == 0 && NT % 32 == 0), SyncWarp, SyncBlock>::type;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int t = threadIdx.x, ly = threadIdx.y;
  const int line = blockIdx.x * blockDim.y + ly;
  const bool valid = line < nlines;
  C* sm = reinterpret_cast<C*>(smem_raw) + ly * zplain_stride<H>();
  for (int k = t; k <= H; k += F::TPL) sm[k] = (valid && k < kin) ? op.load(line, k) : mkc<T>(T(0), T(0));
  if constexpr (sizeof(T) == 8) {
    const int xs = c2r_line_to_fx<H, F::TPL>(sm, H + 1, t, ly, SYNC{});
    longlong2* sx = reinterpret_cast<longlong2*>(sm);
    c2r_line_fx<F, H>(sx, H + 1, sx, t, twH, twM, SYNC{});
    if (valid) {
#pragma unroll 2
      for (int i = 0; i < F::E; ++i) op.store_pair(line, t + i * F::TPL, fx::to_c(sx[pidx<F::kLayout>(t + i * F::TPL)], xs));
    }
    return;
  }
  SYNC{}();
  C v[F::E];
#pragma unroll
  for (int s = 0; s < F::E; ++s) v[s] = c2r_pre<T, H>(sm, F::in_index(t, s), twM);
  F::run(v, t, sm, 1, twH, SYNC{});
  if (valid) {
#pragma unroll
    for (int s = 0; s < F::E; ++s) op.store_pair(line, F::out_index(t, s), v[s]);
  }
}

// ---------------------------------------------------------------------------
// z pass c2r of the three displacement / velocity components of a line, with
// the lattice readout fused (set_positions / set_velocities,
// particle_generator.hh:499-639): particle ip = ishift*n^3 + cell, AoS
// [ip][3] of q + Psi (FP64 sum, stored as P) or, in fields mode, three n^3
// grids of doubles.  Inputs: the three component grids after their x and y
// passes, [line][n/2+1] complex.
// ---------------------------------------------------------------------------
// the lattice readout of cells 2m, 2m+1 of a transformed line (particle
// ip = ishift*n^3 + cell), v the unnormalised component values
template <typename T, typename P>
__device__ __forceinline__ void lattice_out(const Lattice3Args& a, int line, int m, const cplx<T> (&v)[3]) {
  const int n = a.n;
  const long long n3 = (long long)n * n * n;
  const int i = line / n, j = line % n;
  if constexpr (std::is_same<P, float>::value && std::is_same<T, float>::value) {
    if (!a.fields_mode) {
      // FP32 particles: the two particles are 24 contiguous bytes (8-byte
      // aligned for even n), stored as three float2; positions q + Psi with q
      // as a float pair: the correctly rounded sum on the FP32 pipes (ff_add_q)
      float w[6];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int k = 2 * m + h;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const float x = (h ? v[d].y : v[d].x) * T(a.norm);
          const int qi = (d == 0) ? i : ((d == 1) ? n + j : 2 * n + k);
          w[3 * h + d] = a.with_q ? ff_add_q(a.qf[qi], x) : x;
        }
      }
      float2* o = reinterpret_cast<float2*>(reinterpret_cast<float*>(a.dst) +
                                            3 * ((long long)a.ishift * n3 + (long long)line * n + 2 * m));
      o[0] = make_float2(w[0], w[1]);
      o[1] = make_float2(w[2], w[3]);
      o[2] = make_float2(w[4], w[5]);
      return;
    }
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int k = 2 * m + h;
    const long long c = (long long)line * n + k;
    if (std::is_same<P, T>::value && !a.with_q && !a.fields_mode) {
      // velocities (no lattice coordinate) in the grid precision: no FP64 step
      P* o = reinterpret_cast<P*>(a.dst) + 3 * ((long long)a.ishift * n3 + c);
#pragma unroll
      for (int d = 0; d < 3; ++d) o[d] = (P)((h ? v[d].y : v[d].x) * T(a.norm));
      continue;
    }
    double val[3];
    // normalised in the grid precision, as the component grids of the per-component path
#pragma unroll
    for (int d = 0; d < 3; ++d) val[d] = (double)((h ? v[d].y : v[d].x) * T(a.norm));
    if (a.fields_mode) {
      double* o = reinterpret_cast<double*>(a.dst);
#pragma unroll
      for (int d = 0; d < 3; ++d) o[d * n3 + c] = val[d];
    } else {
      if (a.with_q) {
        val[0] += a.q[i];
        val[1] += a.q[n + j];
        val[2] += a.q[2 * n + k];
      }
      P* o = reinterpret_cast<P*>(a.dst) + 3 * ((long long)a.ishift * n3 + c);
#pragma unroll
      for (int d = 0; d < 3; ++d) o[d] = (P)val[d];
    }
  }
}

// Whether the lattice z pass goes component by component through the staged
// lines (one register set) instead of holding three: FP64, and lengths of more
// than eight values per thread.  One staging buffer then, for the warps that
// fit an SM by shared memory.
template <typename T, int H>
__host__ __device__ constexpr bool lattice_staged() {
  return sizeof(T) == 8 || LineFFT<T, H, true>::E > 8;
}
template <typename T, int H, int LPB, typename P>
__global__ void __launch_bounds__(LPB * LineFFT<T, H, true>::TPL, (LineFFT<T, H, true>::E <= 8) ? 2 : 1)
    k_zc2r3_lattice(Lattice3Args a, const cplx<T>* __restrict__ twH, const cplx<T>* __restrict__ twM) {
  // each line's exchanges run in its own staged region (XOR layout of the
  // contiguous-line passes), under warp barriers when a line's threads sit
  // inside one warp; the staged lines of a component are H+1 elements apart,
  // so the line groups take lines TPL apart (zline_of_group).  The layout may
  // not need more than H+1 elements.
  constexpr int LAY = padded_len(H, zlayout(H)) <= H + 1 ? zlayout(H) : 0;
  using F = LineFFT<T, H, true, 8, LAY>;
  using SYNC = typename std::conditional<(F::TPL <= 32 && 32 % F::TPL == 0 && (LPB * F::TPL) % 32 == 0), SyncWarp,
                                         SyncBlock>::type;
  using C = cplx<T>;
  constexpr bool STAGED = lattice_staged<T, H>();
  constexpr int SL = 3 * (H + 1);  // complex values of one line's three components
  // persistent CTAs over batches of LPB lines; in the unstaged form the next
  // batch is copied into the other shared-memory buffer (cp.async) while this
  // one is transformed
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf0 = reinterpret_cast<C*>(smem_raw);
  [[maybe_unused]] C* buf1 = buf0 + LPB * SL;
  const int t = threadIdx.x, lg = threadIdx.y;
  constexpr int WF = 128 / (int)sizeof(C);
  int ly = lg;
  if constexpr (zline_map_ok<F::TPL, WF>(LPB)) ly = zline_of_group<F::TPL, WF>(lg);
  const int tid = lg * F::TPL + t;
  const int Kz = H + 1;
  const int nb = (a.nlines + LPB - 1) / LPB;
  // a batch of one component is LPB consecutive lines, contiguous in global
  // memory: staged as [d][l][k] with 16-byte copies (an even LPB keeps both
  // ends 16-byte aligned)
  static_assert(LPB % 2 == 0, "even lines per batch");
  constexpr int U = LPB * Kz * (int)sizeof(C) / 16;  // 16-byte units per component
  auto issue = [&](int bt, C* buf) {  // nlines is a multiple of LPB (checked at launch)
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const void* base = (d == 0) ? a.comp[0] : ((d == 1) ? a.comp[1] : a.comp[2]);
      const char* g = reinterpret_cast<const char*>(base) + (size_t)bt * LPB * Kz * sizeof(C);
      char* sb = reinterpret_cast<char*>(buf + d * LPB * Kz);
      for (int u = tid; u < U; u += LPB * F::TPL) cp_async16(sb + 16 * u, g + 16 * u);
    }
    cp_async_commit();
  };
  if constexpr (STAGED) {
    for (int bt = blockIdx.x; bt < nb; bt += gridDim.x) {
      issue(bt, buf0);
      cp_async_wait<0>();
      __syncthreads();  // every thread's copies of this batch have landed
      [[maybe_unused]] int xs[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        C* sm = buf0 + d * LPB * Kz + ly * Kz;
        if constexpr (sizeof(T) == 8) xs[d] = c2r_line_to_fx<H, F::TPL>(sm, Kz, t, lg, SYNC{});
      }
#pragma unroll 1
      for (int d = 0; d < 3; ++d) {
        C* sm = buf0 + d * LPB * Kz + ly * Kz;
        if constexpr (sizeof(T) == 8) {
          longlong2* sx = reinterpret_cast<longlong2*>(sm);
          c2r_line_fx<F, H>(sx, Kz, sx, t, twH, twM, SYNC{});
        } else {
          C v[F::E];
#pragma unroll
          for (int s = 0; s < F::E; ++s) v[s] = c2r_pre<T, H>(sm, F::in_index(t, s), twM);
          F::run(v, t, sm, 1, twH, SYNC{});
          SYNC{}();
#pragma unroll
          for (int s = 0; s < F::E; ++s) sm[F::out_slot(t, s)] = v[s];
        }
      }
      // every thread reads back the elements that it wrote
#pragma unroll 2
      for (int q = 0; q < F::E; ++q) {
        const int m = t + q * F::TPL;
        C v[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const C r = buf0[d * LPB * Kz + ly * Kz + pidx<LAY>(m)];
          if constexpr (sizeof(T) == 8) v[d] = fx::to_c(reinterpret_cast<const longlong2&>(r), xs[d]);
          else v[d] = r;
        }
        lattice_out<T, P>(a, bt * LPB + ly, m, v);
      }
      __syncthreads();  // the buffer is refilled by the next iteration's copies
    }
    return;
  } else {
    int bt = blockIdx.x;
    if (bt < nb) issue(bt, buf0); else cp_async_commit();
    for (int it = 0; bt < nb; bt += gridDim.x, ++it) {
      C* cur = (it & 1) ? buf1 : buf0;
      C* nxt = (it & 1) ? buf0 : buf1;
      const int bn = bt + gridDim.x;
      if (bn < nb) issue(bn, nxt); else cp_async_commit();
      cp_async_wait<1>();
      __syncthreads();  // every thread's copies of this batch have landed
      C* sm[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) sm[d] = cur + d * LPB * Kz + ly * Kz;
      C v[3][F::E];
#pragma unroll
      for (int d = 0; d < 3; ++d)
#pragma unroll
        for (int s = 0; s < F::E; ++s) v[d][s] = c2r_pre<T, H>(sm[d], F::in_index(t, s), twM);
#pragma unroll
      for (int d = 0; d < 3; ++d) F::run(v[d], t, sm[d], 1, twH, SYNC{});
#pragma unroll
      for (int s = 0; s < F::E; ++s) {
        const C w[3] = {v[0][s], v[1][s], v[2][s]};
        lattice_out<T, P>(a, bt * LPB + ly, F::out_index(t, s), w);
      }
      __syncthreads();  // cur is refilled by the next iteration's copies
    }
    cp_async_wait<0>();
  }
}

// ---------------------------------------------------------------------------
// fused Orszag z pass: per line, c2r of nop operands, pointwise product of
// the real values, r2c of the product, store of kz in [0, kout)
// ---------------------------------------------------------------------------

// c2r pre-processing read straight from global memory: Z[k] = E + i O with
// A = X[k], B = conj(X[H-k]) (zero for kz >= kin), imaginary parts of the
// kz = 0 and kz = H terms dropped (FFTW's c2r convention)
template <typename T, int H>
__device__ __forceinline__ cplx<T> c2r_pre_g(const cplx<T>* __restrict__ src, int k, int kin,
                                             const cplx<T>* __restrict__ twM) {
  using C = cplx<T>;
  C A = (k < kin) ? src[k] : mkc<T>(T(0), T(0));
  C B = (H - k < kin) ? src[H - k] : mkc<T>(T(0), T(0));
  if (k == 0) { A.y = T(0); B.y = T(0); }
  B = cconj(B);
  const C Ev = cadd(A, B);
  const C Ov = cmulc(csub(A, B), twM[k]);
  return mkc<T>(Ev.x - Ov.y, Ev.y + Ov.x);
}

// One thread group of TPL threads per line; when TPL divides 32 every line
// lives inside one warp and all exchanges use warp barriers only.  The
// operands' inverse transforms read their inputs straight from HBM, the
// running product stays in registers, and only the final r2c
// post-processing goes through shared memory once more.
template <typename T, int H, int MAXR, int NT, int MINB, class SYNC>
__global__ void __launch_bounds__(NT, MINB) k_zconv(ZConvArgs<T> a, const cplx<T>* __restrict__ twH,
                                                const cplx<T>* __restrict__ twM) {
  using FI = LineFFT<T, H, true, MAXR>;
  using FF = LineFFT<T, H, false, MAXR>;
  static_assert(FI::E == FF::E && FI::TPL == FF::TPL, "plan mismatch");
  using C = cplx<T>;
  constexpr int E = FI::E, TPL = FI::TPL, LPB = NT / TPL;
  constexpr int LSTRIDE = H + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int t = threadIdx.x % TPL, ly = threadIdx.x / TPL;
  const int line = blockIdx.x * LPB + ly;
  const bool valid = line < a.nlines;
  C* sm = reinterpret_cast<C*>(smem_raw) + ly * LSTRIDE;
  SYNC sync;
  C v[E], prod[E];
  for (int op = 0; op < a.nop; ++op) {
    const C* base = (op == 0) ? a.in[0] : ((op == 1) ? a.in[1] : a.in[2]);
    const C* src = base + (long long)(valid ? line : 0) * a.in_stride;
    const int kin = valid ? a.kin : 0;
#pragma unroll
    for (int s = 0; s < E; ++s) v[s] = c2r_pre_g<T, H>(src, FI::in_index(t, s), kin, twM);
    FI::run(v, t, sm, 1, twH, sync);
    if (op == 0) {
#pragma unroll
      for (int s = 0; s < E; ++s) prod[s] = v[s];
    } else {
#pragma unroll
      for (int s = 0; s < E; ++s) { prod[s].x *= v[s].x; prod[s].y *= v[s].y; }
    }
  }
  // forward transform of the packed product: one exchange into stage-0 order
  sync();
#pragma unroll
  for (int s = 0; s < E; ++s) sm[FI::out_index(t, s)] = prod[s];
  sync();
#pragma unroll
  for (int s = 0; s < E; ++s) v[s] = sm[FF::in_index(t, s)];
  FF::run(v, t, sm, 1, twH, sync);
  sync();
#pragma unroll
  for (int s = 0; s < E; ++s) sm[FF::out_index(t, s)] = v[s];
  sync();
  if (valid) {
    C* dst = a.out + (long long)line * a.out_stride;
    for (int k = t; k < a.kout; k += TPL) {
      const C zk = sm[k % H];
      const C zc = cconj(sm[(H - k) % H]);
      const C Ev = mkc<T>(T(0.5) * (zk.x + zc.x), T(0.5) * (zk.y + zc.y));
      const C Ov = mkc<T>(T(0.5) * (zk.y - zc.y), -T(0.5) * (zk.x - zc.x));
      dst[k] = cscale(cadd(Ev, cmul(twM[k], Ov)), a.out_scale);
    }
  }
}

// ---------------------------------------------------------------------------
// TMA-pipelined fused z pass.  Persistent CTAs walk batches of LPB
// consecutive lines; the operands of the next batch are fetched by bulk
// asynchronous copies (cp.async.bulk, one per operand, completion counted on
// an mbarrier) into the other half of a double buffer while the current batch
// is transformed, so HBM traffic overlaps the FFT work.
// Shared memory: [2 mbarriers | stage[2][nop][LPB][line stride] | exchange[LPB][line stride]],
// the exchange only where the staged lines cannot hold it; FP64 lines, bound by
// the integer pipes, are transformed in place in one stage.
// ---------------------------------------------------------------------------
template <typename T, int H>
__device__ __forceinline__ cplx<T> c2r_pre_s(const cplx<T>* src, int k, int kin, const cplx<T>* __restrict__ twM) {
  using C = cplx<T>;
  C A = (k < kin) ? src[k] : mkc<T>(T(0), T(0));
  C B = (H - k < kin) ? src[H - k] : mkc<T>(T(0), T(0));
  if (k == 0) { A.y = T(0); B.y = T(0); }
  B = cconj(B);
  const C Ev = cadd(A, B);
  const C Ov = cmulc(csub(A, B), twM[k]);
  return mkc<T>(Ev.x - Ov.y, Ev.y + Ov.x);
}

// Output slots of a line FFT held as k = t + TPL a(s): the r2c post-processing
// pairs Z[k] with Z[H - k], which then sits in lane (TPL - t) mod TPL of the
// same line group, slot a' = E - 1 - a (or (E - a) mod E in lane 0), so one
// warp shuffle per slot replaces a shared-memory round trip.
template <class F>
__host__ __device__ constexpr int zslot_a(int s) {
  return s / F::RL + (F::TPL > 0 ? (F::LEN / F::RL) / F::TPL : 0) * (s % F::RL);
}
template <class F>
__host__ __device__ constexpr bool zshfl_post_ok() {
  if (!(F::TPL <= 32 && 32 % F::TPL == 0 && (F::LEN / F::RL) % F::TPL == 0)) return false;
  bool seen[64] = {};
  if (F::E > 64) return false;
  for (int s = 0; s < F::E; ++s) {
    const int a = zslot_a<F>(s);
    if (a < 0 || a >= F::E || seen[a]) return false;
    seen[a] = true;
  }
  return true;
}
template <class F>
__host__ __device__ constexpr int zslot_of(int a) {
  for (int s = 0; s < F::E; ++s)
    if (zslot_a<F>(s) == a) return s;
  return 0;
}

// MODE 0: the fused convolution z pass above.
// MODE 1: the inverse transform of one operand only, its real line (M reals
//         as H packed pairs) stored to out[line * out_stride + m].
// MODE 2: the forward transform of one real line (H packed pairs, kin = H),
//         stored as kz < kout like MODE 0.
// CTAs per SM the FP32 r2c z pass (MODE 2) is compiled for: it exchanges in
// its staged input lines, so four fit by shared memory at 128 registers
// (0 elsewhere: no minimum, the compiler's register choice)
// FP64 (fixed point): 168 registers, 12 warps
template <typename T, int MODE>
__host__ __device__ constexpr int zconv_tma_minb(int threads) {
  if (sizeof(T) != 4) return 65536 / (168 * threads) > 16 ? 16 : (65536 / (168 * threads) > 0 ? 65536 / (168 * threads) : 1);
  return MODE == 2 ? 4 : 0;
}
// the r2c mode exchanges in its staged input lines (kin = H, zstage_stride
// apart) when the exchange stride of a line fits in one
template <int H, int MODE>
__host__ __device__ constexpr bool zconv_xchg_in_stage() {
  return MODE == 2 && zline_stride(H) <= zstage_stride(H);
}
// FP64 lines are staged one by one, zfx_stride elements apart, and transformed
// in place in fixed point
template <int H>
__host__ __device__ constexpr int zfx_stride(int kin) {
  return zline_stride(H) > kin ? zline_stride(H) : kin;
}
template <typename T, int H, int MAXR, int LPB, class SYNC, int MODE = 0, int KIN = 0>
__global__ void __launch_bounds__(LPB * LineFFT<T, H, true, MAXR>::TPL,
                                  zconv_tma_minb<T, MODE>(LPB * LineFFT<T, H, true, MAXR>::TPL))
k_zconv_tma(ZConvArgs<T> a, const cplx<T>* __restrict__ twH, const cplx<T>* __restrict__ twM) {
  constexpr int LAY = zlayout(H);
  using FI = LineFFT<T, H, true, MAXR, LAY, true, sizeof(T) == 8 || MODE != 1 || zinv_split(H)>;
  using FF = LineFFT<T, H, false, MAXR, LAY, true>;
  using C = cplx<T>;
  constexpr int E = FI::E, TPL = FI::TPL;
  constexpr int LS = zline_stride(H);  // per-line exchange length
  extern __shared__ __align__(128) unsigned char smem_raw[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw);
  const int nop = (MODE == 0) ? a.nop : 1;
  const int kin = KIN ? KIN : a.kin;  // line length (compiled in when KIN > 0)
  C* stage = reinterpret_cast<C*>(smem_raw + 128);
  constexpr int SP2 = zstage_stride(H);  // staged line stride of the r2c mode
  constexpr bool PER_LINE = MODE == 2 && SP2 != H;  // its lines are copied one by one
  const int sline = (MODE == 2) ? SP2 : kin;
  const int per_op = LPB * sline;
  C* xchg = stage + 2 * nop * per_op;
  constexpr int WF = 128 / (int)sizeof(C);  // elements per shared-memory wavefront
  const int t = threadIdx.x % TPL, lg = threadIdx.x / TPL;
  int ly = lg;
  if constexpr (MODE != 2 && zline_map_ok<TPL, WF>(LPB)) ly = zline_of_group<TPL, WF>(lg);
  C* const sm_x = xchg + lg * LS;
  const int nbatch = a.nlines / LPB;
  const unsigned bytes_op = (unsigned)(LPB * kin * sizeof(C));
  const C* in0 = a.in[0];
  const C* in1 = a.in[1];
  const C* in2 = a.in[2];
  SYNC sync;
  if (threadIdx.x == 0) {
    mbar_init(&bars[0], 1);
    mbar_init(&bars[1], 1);
    fence_mbar_init();
  }
  __syncthreads();
  if constexpr (sizeof(T) == 8) {
    // One buffer per CTA: the pass is bound by the integer pipes, and smaller
    // CTAs fill the SM better than a second buffer.  The conversions are
    // rolled loops over the staged line (mf_fx.cuh).
    const int sl = zfx_stride<H>(kin);
    const int kx = (MODE == 2) ? H : kin;
    int it = 0;
    for (int b = blockIdx.x; b < nbatch; b += gridDim.x, ++it) {
      if (threadIdx.x < 32) {
        fence_proxy_async_smem();
        if (threadIdx.x == 0) mbar_arrive_expect_tx(&bars[0], (unsigned)(nop * LPB * kx * (int)sizeof(C)));
        __syncwarp();
        for (int l = threadIdx.x; l < nop * LPB; l += 32) {
          const int op = l / LPB, ln = l - op * LPB;
          const C* in = (op == 0) ? in0 : ((op == 1) ? in1 : in2);
          tma_load_1d(stage + l * sl, in + ((long long)b * LPB + ln) * kx, (unsigned)(kx * sizeof(C)), &bars[0]);
        }
      }
      const bool ok = mbar_wait_bounded(&bars[0], it & 1, a.err, 1);
      if (!__syncthreads_and(ok)) return;
      C* dst = a.out + (long long)(b * LPB + lg) * a.out_stride;
      C* const l0 = stage + lg * sl;
      if constexpr (MODE != 2) {
        const int nops = (MODE == 0) ? nop : 1;
#pragma unroll 1
        for (int op = 0; op < nops; ++op) {
          C* src = stage + (op * LPB + lg) * sl;
          longlong2* xl = reinterpret_cast<longlong2*>(src);
          const int xs = c2r_line_to_fx<H, TPL>(src, kin, t, lg, sync);
          c2r_line_fx<FI, H>(xl, kin, xl, t, twH, twM, sync);
          // (a thread reads back the elements that it wrote)
          if (MODE == 0) sync();  // the product goes into the first line in another order
#pragma unroll 2
          for (int i = 0; i < E; ++i) {
            const int m = t + i * TPL;
            const C r = fx::to_c(xl[pidx<LAY>(m)], xs);
            if (MODE == 1) dst[m] = r;
            else l0[pidx<LAY>(m)] = (op == 0) ? r : mkc<T>(l0[pidx<LAY>(m)].x * r.x, l0[pidx<LAY>(m)].y * r.y);
          }
        }
      }
      if constexpr (MODE != 1) {
        constexpr int LIN = (MODE == 0) ? LAY : 0;  // layout of the real-space line
        longlong2* xl = reinterpret_cast<longlong2*>(l0);
        const int xs = r2c_line_to_fx<H, TPL, LIN>(l0, t, lg, sync);
        r2c_line_fx<FF, H, LIN>(xl, xl, t, twH, sync);
        const bool unit = a.out_scale == T(1);
#pragma unroll 2
        for (int k = t; k < a.kout; k += TPL) {
          const C r = r2c_line_out<H, LAY>(xl, k, xs, twM);
          dst[k] = unit ? r : cscale(r, a.out_scale);
        }
      }
      __syncthreads();  // the stage is read: the next batch may land in it
    }
    return;
  }
  // run by the first warp
  auto issue = [&](int b, int st) {
    const long long off = (long long)b * LPB * kin;
    if constexpr (PER_LINE) {
      if (threadIdx.x == 0) mbar_arrive_expect_tx(&bars[st], bytes_op);
      __syncwarp();
      for (int l = threadIdx.x; l < LPB; l += 32)
        tma_load_1d(stage + st * per_op + l * SP2, in0 + off + (long long)l * H, (unsigned)(H * sizeof(C)), &bars[st]);
      return;
    }
    if (threadIdx.x != 0) return;
    mbar_arrive_expect_tx(&bars[st], (unsigned)nop * bytes_op);
    tma_load_1d(stage + (st * nop + 0) * per_op, in0 + off, bytes_op, &bars[st]);
    if (nop > 1) tma_load_1d(stage + (st * nop + 1) * per_op, in1 + off, bytes_op, &bars[st]);
    if (nop > 2) tma_load_1d(stage + (st * nop + 2) * per_op, in2 + off, bytes_op, &bars[st]);
  };
  if (threadIdx.x < 32 && (int)blockIdx.x < nbatch) issue(blockIdx.x, 0);
  int iter = 0;
  bool pending_other = false;
  for (int b = blockIdx.x; b < nbatch; b += gridDim.x, ++iter) {
    const int st = iter & 1;
    const int bn = b + gridDim.x;
    if (threadIdx.x < 32 && bn < nbatch) {
      fence_proxy_async_smem();
      issue(bn, st ^ 1);
    }
    pending_other = bn < nbatch;
    const bool ok = mbar_wait_bounded(&bars[st], (iter >> 1) & 1, a.err, 1);
    if (!__syncthreads_and(ok)) {
      // give the copy still in flight into the other buffer a bounded chance to land
      if (pending_other) mbar_wait_bounded(&bars[st ^ 1], ((iter + 1) >> 1) & 1, nullptr, 0);
      return;
    }
    C v[E], prod[E];
    // this line's exchange area: its staged input line in the r2c mode (read
    // into registers before the transform's first exchange), else its own
    C* const sm = zconv_xchg_in_stage<H, MODE>() ? stage + (st * nop) * per_op + ly * sline : sm_x;
    if constexpr (MODE == 2) {
      const C* src = stage + (st * nop) * per_op + ly * sline;
#pragma unroll
      for (int s = 0; s < E; ++s) v[s] = src[FF::in_index(t, s)];
    }
    const int nops = (MODE == 0) ? nop : (MODE == 1 ? 1 : 0);  // compile-time for the one-transform modes
    for (int op = 0; op < nops; ++op) {
      const C* src = stage + (st * nop + op) * per_op + ly * kin;
#pragma unroll
      for (int s = 0; s < E; ++s) v[s] = c2r_pre_s<T, H>(src, FI::in_index(t, s), kin, twM);
      FI::run(v, t, sm, 1, twH, sync);
      if (op == 0) {
#pragma unroll
        for (int s = 0; s < E; ++s) prod[s] = v[s];
      } else {
#pragma unroll
        for (int s = 0; s < E; ++s) { prod[s].x *= v[s].x; prod[s].y *= v[s].y; }
      }
    }
    if constexpr (MODE == 1) {
      C* dst = a.out + (long long)(b * LPB + ly) * a.out_stride;
#pragma unroll
      for (int s = 0; s < E; ++s) dst[FI::out_index(t, s)] = prod[s];
    } else {
      if constexpr (MODE == 0) {
        sync();
#pragma unroll
        for (int s = 0; s < E; ++s) sm[FI::out_slot(t, s)] = prod[s];
        sync();
#pragma unroll
        for (int s = 0; s < E; ++s) v[s] = sm[FF::in_slot(t, s)];
      }
      FF::run(v, t, sm, 1, twH, sync);
      C* dst = a.out + (long long)(b * LPB + ly) * a.out_stride;
      if constexpr (zshfl_post_ok<FF>()) {
        // Z[H - k] from the partner lane by shuffles (no exchange through shared memory)
        const int lane = threadIdx.x & 31;
        const int src = (lane & ~(TPL - 1)) + ((TPL - t) & (TPL - 1));
        // slots that can hold a kept k: the r2c mode keeps kz <= 2H/3 (the
        // Orszag N/2, checked at launch), the fused pass up to H
        constexpr int QK = (MODE == 2) ? (2 * H / 3 + 1 + TPL - 1) / TPL : E;
        constexpr int QMAX = QK < E ? QK : E;
#pragma unroll
        for (int q = 0; q < QMAX; ++q) {
          const C give = (t == 0) ? v[zslot_of<FF>((E - q) % E)] : v[zslot_of<FF>(E - 1 - q)];
          C zc;
          zc.x = __shfl_sync(0xffffffffu, give.x, src);
          zc.y = -__shfl_sync(0xffffffffu, give.y, src);
          const int k = t + TPL * q;
          const C zk = v[zslot_of<FF>(q)];
          if (k < a.kout) {
            const C Ev = mkc<T>(T(0.5) * (zk.x + zc.x), T(0.5) * (zk.y + zc.y));
            const C Ov = mkc<T>(T(0.5) * (zk.y - zc.y), -T(0.5) * (zk.x - zc.x));
            dst[k] = cscale(cadd(Ev, cmul(twM[k], Ov)), a.out_scale);
          }
        }
        if (t == 0 && a.kout > H) {  // k = H (kept when kout = H + 1): Z[H] = Z[0]
          const C zk = v[zslot_of<FF>(0)];
          const C Ev = mkc<T>(zk.x, T(0));
          const C Ov = mkc<T>(zk.y, T(0));
          dst[H] = cscale(cadd(Ev, cmul(twM[H], Ov)), a.out_scale);
        }
        __syncthreads();  // stage[st] fully consumed before it is refilled
        continue;
      }
      sync();
#pragma unroll
      for (int s = 0; s < E; ++s) sm[pidx<LAY>(FF::out_index(t, s))] = v[s];
      sync();
      for (int k = t; k < a.kout; k += TPL) {
        const C zk = sm[pidx<LAY>(k % H)];
        const C zc = cconj(sm[pidx<LAY>((H - k) % H)]);
        const C Ev = mkc<T>(T(0.5) * (zk.x + zc.x), T(0.5) * (zk.y + zc.y));
        const C Ov = mkc<T>(T(0.5) * (zk.y - zc.y), -T(0.5) * (zk.x - zc.x));
        dst[k] = cscale(cadd(Ev, cmul(twM[k], Ov)), a.out_scale);
      }
    }
    __syncthreads();  // stage[st] fully consumed before it is refilled
  }
}

}  // namespace mf
