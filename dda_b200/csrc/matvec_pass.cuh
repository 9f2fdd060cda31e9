// matvec_pass.cuh -- the y/z passes of the matvec as three kernels over a
// bounded work buffer:
//
//   k_zfwd   forward FFT along z of column tiles of the kx planes,
//   k_rows   per (kx, kz) row: forward FFT along y, D-hat multiply, inverse
//            FFT along y,
//   k_zinv   inverse FFT along z, back to the planes.
//
// k_yz_p keeps a whole plane in one CTA's shared memory, so an SM holds one
// CTA of 16 warps whose stages all end at its barriers.  Here a CTA holds a
// column tile (256 bytes of every kz: 2 KB at Gz = 8, 64 KB at 256; half of that
// beyond) or a few rows (up to 48 KB, see RTile), with the twiddles and in the
// row kernel a D-hat row beside them; an SM holds several CTAs in different
// phases, and every global access is the first or last butterfly
// stage of a line: inputs go from HBM or L2 to registers, outputs from
// registers back, and each transform passes through shared memory K - 1
// times for a K-stage plan.
//
// W = 2 (FP32): the transforms of two right-hand sides run side by side as
// P2 values, each operation one two-lane instruction, with shared twiddles,
// D-hat loads and index arithmetic.  W = 1: one right-hand side.  The lanes
// are rounded alike, so a right-hand side has the same bits either way.
//
// What bounds them and what they take (16 right-hand sides of the spheroid,
// planes 128 x 128 with by = bz = 64, FP32, W = 2; HBM floor at 6.5 TB/s): z
// forward 148 us and z inverse 154 us of 140 us (HBM); rows 395 us of 188 us,
// with the FMA pipe busy 56 % of the time, the shared-memory pipe 65 %, and
// 13 warps an SM (128 registers) to cover the latency between the two.  The
// plane kernel took 1 202 us for all of it; 128 right-hand sides 9.41 -> 5.39 ms,
// 512^3 (two) 12.9 -> 6.5 ms (cluster kernel).  W = 1 instead of 2: rows 424
// us.  Twiddles from global memory through L1 instead of shared memory: rows
// 492 us, z forward 182 us.
//
// The work buffer holds zbuf[pair][plane][kz][3 by] of a chunk of planes:
// plane 2 i + f is frequency kx = ax0 + i (f = 0) or its mirror Gx - kx
// (f = 1), kz in frequency order.  A CTA of k_rows takes the four mirrored
// rows (+-kx, +-kz) of one D-hat octant row, or fewer of them where rows are
// long, and loads the octant row once.
#pragma once

#include <algorithm>

#include "fft_plan.cuh"
#include "matvec_kernels.cuh"
#include "matvec_planned.cuh"

namespace dda {

// Twiddles of plan P's stage I in butterfly-major order: entry
// StageTw<P>::off(I) + (m - 1) S + j = exp(-2 pi i j m / L), m in [1, R).
template <typename P> struct StageTw {
  static __host__ __device__ constexpr int off(int i) {
    int o = 0;
    for (int k = 0; k < i; k++) o += (P::r[k] - 1) * (P::L(k) / P::r[k]);
    return o;
  }
  static __host__ __device__ constexpr int count() { return (off(P::K - 1) + 1) / 2 * 2; }  // even: 16-byte aligned
};

// Value type of W right-hand sides in precision T.
template <typename T, int W> struct PassV { typedef typename C2<T>::t t; };
template <> struct PassV<float, 2> { typedef P2 t; };

// Shared-memory position of element p of a line whose blocks of the last
// radix are padded to an odd pitch: neighbouring threads that take
// neighbouring blocks then hit different banks.
template <typename P> struct RowPad {
  enum : int { RL = P::r[P::K - 1], RP = RL | 1, S0 = P::N / P::r[0] };
  static __host__ __device__ constexpr int at(int p) { return p / RL * RP + p % RL; }
  // line pitch for elements of `bytes`: congruent to the first stage's
  // butterflies modulo the elements of 128 bytes, so that the items of
  // consecutive lines continue one another's banks
  static __host__ __device__ constexpr int pitch(int bytes) {
    const int mod = 128 / bytes;
    int lp = P::N / RL * RP;
    while (lp % mod != S0 % mod) lp++;
    return lp;
  }
};

template <typename P, int I, bool INV, typename V, typename W>
__device__ __forceinline__ void pass_twiddle(V* v, int j, const W* tw) {
  constexpr int R = P::r[I], S = P::L(I) / R;
  constexpr int O = StageTw<P>::off(I);
#pragma unroll
  for (int m = 1; m < R; m++) {
    W w = tw[O + (m - 1) * S + j];
    if (INV) w.y = -w.y;
    v[m] = cmul(v[m], w);
  }
}

// Copies plan P's stage twiddles to shared memory (asynchronously; wait with
// pass_tw_wait and a barrier).
template <typename P, typename W>
__device__ __forceinline__ void pass_tw_copy(W* dst, const W* __restrict__ src) {
  constexpr int N16 = StageTw<P>::count() * (int)sizeof(W) / 16;
  for (int i = threadIdx.x; i < N16; i += blockDim.x)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(
                     reinterpret_cast<float4*>(dst) + i)),
                 "l"(reinterpret_cast<const float4*>(src) + i));
}
__device__ __forceinline__ void pass_tw_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Frequency of position t R_last (its blocks' first element): element m of
// the block holds that frequency + m N / R_last.
template <typename P> __device__ __forceinline__ int block_freq(int t) {
  constexpr int RL = P::r[P::K - 1];
  return P::freq_of(t * RL);
}

struct PassGeom {
  int Gx, Gy, Gz, by, bz, nb;  // nb = by bz
  int b0, nrhs;                // right-hand sides [b0, nrhs) of this launch, W per work-buffer entry
  int ax0, nax;                // frequencies [ax0, ax0 + nax) of this chunk
  const int* xpos;             // frequency -> position along x
};

// Plane of work-buffer index pl: its position along x, -1 for the mirror of
// a frequency that is its own.
__device__ __forceinline__ int pass_plane(const PassGeom& p, int pl) {
  const int ax = p.ax0 + (pl >> 1), f = pl & 1;
  if (f && (ax == 0 || 2 * ax == p.Gx)) return -1;
  return p.xpos[f ? p.Gx - ax : ax];
}

// Right-hand sides of entry w: first and whether each of them runs.
template <int W>
struct PassRhs {
  int b;
  bool on0, on1;
  __device__ __forceinline__ PassRhs(const PassGeom& p, int w, const KrylovState* st, int mvskip) {
    b = p.b0 + w * W;
    on0 = !rhs_idle(st, b, mvskip);
    on1 = W == 2 && b + 1 < p.nrhs && !rhs_idle(st, b + 1, mvskip);
  }
  __device__ __forceinline__ bool any() const { return on0 || on1; }
};

__device__ __forceinline__ float2 pass_ld(const float2* a) { return __ldcs(a); }
__device__ __forceinline__ double2 pass_ld(const double2* a) { return __ldcs(a); }

// One middle stage (1 <= I < K - 1) of NL lines, in place.  at(l, p): shared
// address of element p of line l; items with the line fastest when COL.
template <typename P, int I, bool INV, typename V, typename W, bool COL, int NT, typename At>
__device__ __forceinline__ void pass_middle(V* sm, int nl, const W* tw, At at) {
  constexpr int R = P::r[I], L = P::L(I), S = L / R, NB = P::N / R;
  for (int it = threadIdx.x; it < nl * NB; it += NT) {
    const int t = COL ? it / nl : it % NB, l = COL ? it - t * nl : it / NB;
    const int blk = t / S, j = t - blk * S;
    V v[R];
#pragma unroll
    for (int m = 0; m < R; m++) v[m] = sm[at(l, blk * L + j + m * S)];
    if (INV) pass_twiddle<P, I, true>(v, j, tw);
    DftN<R, INV, V>::run(v);
    if (!INV) pass_twiddle<P, I, false>(v, j, tw);
#pragma unroll
    for (int m = 0; m < R; m++) sm[at(l, blk * L + j + m * S)] = v[m];
  }
  __syncthreads();
}
template <typename P, bool INV, int I0, int I1, typename V, typename W, bool COL, int NT, typename At>
__device__ __forceinline__ void pass_middles(V* sm, int nl, const W* tw, At at) {
  if constexpr (I0 < I1) {
    if constexpr (!INV) {
      pass_middle<P, I0, false, V, W, COL, NT>(sm, nl, tw, at);
      pass_middles<P, INV, I0 + 1, I1, V, W, COL, NT>(sm, nl, tw, at);
    } else {
      pass_middle<P, I1 - 1, true, V, W, COL, NT>(sm, nl, tw, at);
      pass_middles<P, INV, I0, I1 - 1, V, W, COL, NT>(sm, nl, tw, at);
    }
  }
}

// Threads for `items` work items: as few rounds of at most 256 threads as
// they need, evenly filled.
__host__ __device__ constexpr int pass_threads(int items, int most = 256) {
  const int rounds = (items + most - 1) / most;
  return ((items + rounds - 1) / rounds + 31) / 32 * 32;
}
// CTAs an SM must hold for at most `regs` registers per thread.
__host__ __device__ constexpr int pass_ctas(int nt, int regs) { return 65536 / (nt * regs) > 0 ? 65536 / (nt * regs) : 1; }

// Column tiles of k_zfwd / k_zinv: a row segment of 256 bytes, 128 where the
// tile would take more than 64 KB and an SM hold one or two CTAs (512, two
// right-hand sides, a quarter of the planes: 591 -> 338 us forward; at 128,
// 148 -> 228); one or two first (last) butterflies per thread (inverse at 128
// with 128 threads instead of 256: 156 -> 188 us).
template <typename V, typename P> struct ZTile {
  enum : int {
    SEG = P::N > 256 ? 128 : 256,
    TC = SEG / (int)sizeof(V),
    NTF = pass_threads(TC * (P::N / P::r[0])),
    NTI = pass_threads(TC * (P::N / P::r[P::K - 1])),
    REGS = sizeof(V) == 16 ? 128 : 80,
    CTF = pass_ctas(NTF, REGS),
    CTI = pass_ctas(NTI, REGS)
  };
};

// Rows per CTA of k_rows (of the four mirrored ones) and its threads: all four
// while they take at most 48 KB, so that four to seven CTAs share an SM (160:
// four rows 79.5 us, two 90.4; 512: one row 974 us, four 2 400).  Registers per
// thread: as many as leave the most warps without spills that cost more (FP64,
// 16 x 8: 128 registers 482 us, 160 438; 20 x 5: 89 and 95; P2, 16 x 8: 383 and
// 407; FP32, 32 x 8: 80 registers 296 us, 96 286).  Measured at these plans;
// others take the limit of the nearest, and in FP64 30 x 6 and 30 x 7 spill 152
// bytes at 128, as k_zfwd does 112 to 160 with first radices of 30 and 32.
template <typename V, typename P> struct RTile {
  enum : int {
    LINE = 3 * RowPad<P>::pitch(sizeof(V)) * (int)sizeof(V),
    RQ = LINE <= 12288 ? 4 : LINE <= 20480 ? 2 : 1,
    IT0 = RQ * 3 * (P::N / P::r[0]),
    IT1 = RQ * (P::N / P::r[P::K - 1]),
    NT = pass_threads(P::K == 2 ? IT1 : IT0, 128),
    REGS = std::is_same<V, double2>::value ? (P::K == 2 && P::r[P::K - 1] == 8 ? 160 : 128)
           : sizeof(V) == 16               ? 128
           : P::r[0] >= 28                 ? 96
                                           : 80,
    CTAS = pass_ctas(NT, REGS)
  };
};

// grid (ceil(3 by / TC), 2 nax, entries); shared memory [Gz][TC] values.
template <typename T, int W, typename PZ>
__global__ void __launch_bounds__(ZTile<typename PassV<T, W>::t, PZ>::NTF, ZTile<typename PassV<T, W>::t, PZ>::CTF)
    k_zfwd(const typename C2<T>::t* __restrict__ xhat, typename PassV<T, W>::t* __restrict__ zbuf, PassGeom p,
           const typename C2<T>::t* __restrict__ twg, const KrylovState* __restrict__ st, int mvskip) {
  typedef typename C2<T>::t T2;
  typedef typename PassV<T, W>::t V;
  constexpr int TC = ZTile<V, PZ>::TC, NT = ZTile<V, PZ>::NTF, K = PZ::K, R = PZ::r[0], S0 = PZ::N / R, NZ = (R + 1) / 2;
  const int kx = pass_plane(p, blockIdx.y);
  const PassRhs<W> rh(p, blockIdx.z, st, mvskip);
  if (kx < 0 || !rh.any()) return;
  T2* tw = reinterpret_cast<T2*>(dda_smem);
  V* sm = reinterpret_cast<V*>(tw + StageTw<PZ>::count());
  pass_tw_copy<PZ>(tw, twg);
  const int w3 = 3 * p.by, l0 = blockIdx.x * TC;
  const size_t pstride = (size_t)p.Gx * 3 * p.nb;
  const T2* plane = xhat + ((size_t)rh.b * p.Gx + kx) * 3 * p.nb;
  for (int i0 = 0; i0 < TC * S0; i0 += NT) {
    const int it = i0 + threadIdx.x, l = it % TC, j = it / TC, gl = l0 + l;
    const bool on = it < TC * S0 && gl < w3;
    V v[R];
    if (on) {
      const int c = gl / p.by;
      const T2* src = plane + (size_t)c * p.nb + (gl - c * p.by);
#pragma unroll
      for (int m = 0; m < NZ; m++) {
        const int z = j + m * S0;
        if constexpr (W == 1) {
          v[m] = z < p.bz ? pass_ld(src + (size_t)z * p.by) : czero<V>();
        } else {
          const T2 a = z < p.bz && rh.on0 ? pass_ld(src + (size_t)z * p.by) : czero<T2>();
          const T2 b = z < p.bz && rh.on1 ? pass_ld(src + pstride + (size_t)z * p.by) : czero<T2>();
          v[m].r = make_float2(a.x, b.x);
          v[m].i = make_float2(a.y, b.y);
        }
      }
    }
    if (i0 == 0) {
      pass_tw_wait();
      __syncthreads();
    }
    if (on) {
      DftN<R, false, V, NZ>::run(v);
      pass_twiddle<PZ, 0, false>(v, j, tw);
#pragma unroll
      for (int m = 0; m < R; m++) sm[(j + m * S0) * TC + l] = v[m];
    }
  }
  __syncthreads();
  pass_middles<PZ, false, 1, K - 1, V, T2, true, NT>(sm, TC, tw, [](int l, int q) { return q * TC + l; });
  constexpr int RL = PZ::r[K - 1], NB = PZ::N / RL;
  V* out = zbuf + ((size_t)blockIdx.z * gridDim.y + blockIdx.y) * p.Gz * w3 + l0;
  for (int it = threadIdx.x; it < TC * NB; it += NT) {
    const int l = it % TC, t = it / TC;
    if (l0 + l < w3) {
      V v[RL];
#pragma unroll
      for (int m = 0; m < RL; m++) v[m] = sm[(t * RL + m) * TC + l];
      DftN<RL, false, V>::run(v);
      const int kz = block_freq<PZ>(t);
#pragma unroll
      for (int m = 0; m < RL; m++) out[(size_t)(kz + m * NB) * w3 + l] = v[m];
    }
  }
}

// The inverse: same grid, tile and shared memory.
template <typename T, int W, typename PZ>
__global__ void __launch_bounds__(ZTile<typename PassV<T, W>::t, PZ>::NTI, ZTile<typename PassV<T, W>::t, PZ>::CTI)
    k_zinv(typename C2<T>::t* __restrict__ xhat, const typename PassV<T, W>::t* __restrict__ zbuf, PassGeom p,
           const typename C2<T>::t* __restrict__ twg, const KrylovState* __restrict__ st, int mvskip) {
  typedef typename C2<T>::t T2;
  typedef typename PassV<T, W>::t V;
  constexpr int TC = ZTile<V, PZ>::TC, NT = ZTile<V, PZ>::NTI, K = PZ::K, R = PZ::r[0], S0 = PZ::N / R, NZ = (R + 1) / 2;
  const int kx = pass_plane(p, blockIdx.y);
  const PassRhs<W> rh(p, blockIdx.z, st, mvskip);
  if (kx < 0 || !rh.any()) return;
  T2* tw = reinterpret_cast<T2*>(dda_smem);
  V* sm = reinterpret_cast<V*>(tw + StageTw<PZ>::count());
  pass_tw_copy<PZ>(tw, twg);
  const int w3 = 3 * p.by, l0 = blockIdx.x * TC;
  const size_t pstride = (size_t)p.Gx * 3 * p.nb;
  T2* plane = xhat + ((size_t)rh.b * p.Gx + kx) * 3 * p.nb;
  constexpr int RL = PZ::r[K - 1], NB = PZ::N / RL;
  const V* in = zbuf + ((size_t)blockIdx.z * gridDim.y + blockIdx.y) * p.Gz * w3 + l0;
  for (int it = threadIdx.x; it < TC * NB; it += NT) {
    const int l = it % TC, t = it / TC;
    if (l0 + l < w3) {
      const int kz = block_freq<PZ>(t);
      V v[RL];
#pragma unroll
      for (int m = 0; m < RL; m++) v[m] = in[(size_t)(kz + m * NB) * w3 + l];
      DftN<RL, true, V>::run(v);
#pragma unroll
      for (int m = 0; m < RL; m++) sm[(t * RL + m) * TC + l] = v[m];
    }
  }
  pass_tw_wait();
  __syncthreads();
  pass_middles<PZ, true, 1, K - 1, V, T2, true, NT>(sm, TC, tw, [](int l, int q) { return q * TC + l; });
  for (int it = threadIdx.x; it < TC * S0; it += NT) {
    const int l = it % TC, j = it / TC, gl = l0 + l;
    if (gl < w3) {
      const int c = gl / p.by;
      T2* dst = plane + (size_t)c * p.nb + (gl - c * p.by);
      V v[R];
#pragma unroll
      for (int m = 0; m < R; m++) v[m] = sm[(j + m * S0) * TC + l];
      pass_twiddle<PZ, 0, true>(v, j, tw);
      DftN<R, true, V>::run(v);
#pragma unroll
      for (int m = 0; m < NZ; m++) {
        const int z = j + m * S0;
        if (z < p.bz) {
          if constexpr (W == 1) {
            dst[(size_t)z * p.by] = v[m];
          } else {
            if (rh.on0) dst[(size_t)z * p.by] = make_float2(v[m].r.x, v[m].i.x);
            if (rh.on1) dst[pstride + (size_t)z * p.by] = make_float2(v[m].r.y, v[m].i.y);
          }
        }
      }
    }
  }
}

// Six D-hat components of one point, 16 bytes at a time.
__device__ __forceinline__ void load_d6(const float2* s, float2 d[6]) {
  const float4* q = reinterpret_cast<const float4*>(s);
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const float4 w = q[i];
    d[2 * i] = make_float2(w.x, w.y);
    d[2 * i + 1] = make_float2(w.z, w.w);
  }
}
__device__ __forceinline__ void load_d6(const double2* s, double2 d[6]) {
#pragma unroll
  for (int i = 0; i < 6; i++) d[i] = s[i];
}
// d = -d when f
__device__ __forceinline__ void flip(float2& d, bool f) {
  const unsigned m = f ? 0x80000000u : 0u;
  d.x = __uint_as_float(__float_as_uint(d.x) ^ m);
  d.y = __uint_as_float(__float_as_uint(d.y) ^ m);
}
__device__ __forceinline__ void flip(double2& d, bool f) {
  if (f) { d.x = -d.x; d.y = -d.y; }
}

// Shared memory of k_rows: the D-hat row, the twiddles, RQ rows.
template <typename T, int W, typename PY>
__host__ __device__ constexpr size_t rows_smem() {
  typedef typename PassV<T, W>::t V;
  return (size_t)((PY::N / 2 + 1) * 6 + StageTw<PY>::count()) * sizeof(typename C2<T>::t) +
         (size_t)RTile<V, PY>::RQ * RTile<V, PY>::LINE;
}

// grid ((Gz/2 + 1) 4 / RQ, nax, entries): RQ of the rows (+-kx, +-kz) of one
// entry of the work buffer; RQ = 2: both signs of kz, RQ = 1: one row.
template <typename T, int W, typename PY>
__global__ void __launch_bounds__(RTile<typename PassV<T, W>::t, PY>::NT, RTile<typename PassV<T, W>::t, PY>::CTAS)
    k_rows(typename PassV<T, W>::t* __restrict__ zbuf, const typename C2<T>::t* __restrict__ dc, PassGeom p,
           const typename C2<T>::t* __restrict__ twg, const KrylovState* __restrict__ st, int mvskip) {
  typedef typename C2<T>::t T2;
  typedef typename PassV<T, W>::t V;
  typedef RowPad<PY> Pad;
  constexpr int K = PY::K, N = PY::N, R = PY::r[0], S0 = N / R, NZ = (R + 1) / 2, RL = PY::r[K - 1], NB = N / RL;
  constexpr int LP = Pad::pitch(sizeof(V)), HY = N / 2 + 1;
  constexpr int RQ = RTile<V, PY>::RQ, NT = RTile<V, PY>::NT, PER = 4 / RQ;
  const int az = blockIdx.x / PER, f0 = (blockIdx.x - az * PER) * RQ, ax = p.ax0 + blockIdx.y;
  // row q of this CTA has the signs of f = f0 + q: bit 0 kz, bit 1 kx
  const bool mx = ax != 0 && 2 * ax != p.Gx, mz = az != 0 && 2 * az != p.Gz;
  auto row_on = [&](int q) { const int f = f0 + q; return (mz || !(f & 1)) && (mx || !(f & 2)); };
  if (!PassRhs<W>(p, blockIdx.z, st, mvskip).any()) return;
  if (RQ < 4 && !row_on(0)) return;  // row 0 is off only together with all others
  const int w3 = 3 * p.by;
  auto row_ptr = [&](int q) {
    const int f = f0 + q, pl = 2 * blockIdx.y + (f >> 1), kz = (f & 1) ? p.Gz - az : az;
    return zbuf + (((size_t)blockIdx.z * 2 * p.nax + pl) * p.Gz + kz) * w3;
  };
  T2* sd = reinterpret_cast<T2*>(dda_smem);
  T2* tw = sd + HY * 6;
  V* sm = reinterpret_cast<V*>(tw + StageTw<PY>::count());
  pass_tw_copy<PY>(tw, twg);
  {
    const float4* src = reinterpret_cast<const float4*>(dc + ((size_t)ax * (p.Gz / 2 + 1) + az) * HY * 6);
    float4* dst = reinterpret_cast<float4*>(sd);
    for (int i = threadIdx.x; i < (int)(HY * 6 * sizeof(T2) / 16); i += NT)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst + i)),
                   "l"(src + i));
  }
  for (int i0 = 0; i0 < RQ * 3 * S0; i0 += NT) {
    const int it = i0 + threadIdx.x, j = it % S0, rc = it / S0, q = rc / 3, c = rc - 3 * q;
    const bool on = it < RQ * 3 * S0 && row_on(q);
    V v[R];
    if (on) {
      const V* src = row_ptr(q) + c * p.by;
#pragma unroll
      for (int m = 0; m < NZ; m++) {
        const int y = j + m * S0;
        v[m] = y < p.by ? src[y] : czero<V>();
      }
    }
    if (i0 == 0) {
      pass_tw_wait();
      __syncthreads();
    }
    if (on) {
      DftN<R, false, V, NZ>::run(v);
      pass_twiddle<PY, 0, false>(v, j, tw);
      V* dst = sm + rc * LP + Pad::at(j);
#pragma unroll
      for (int m = 0; m < R; m++) dst[Pad::at(m * S0)] = v[m];
    }
  }
  __syncthreads();
  auto at = [](int l, int q) { return l * LP + Pad::at(q); };
  pass_middles<PY, false, 1, K - 1, V, T2, false, NT>(sm, RQ * 3, tw, at);
  for (int it = threadIdx.x; it < RQ * NB; it += NT) {
    const int t = it % NB, q = it / NB;
    if (!row_on(q)) continue;
    V* s = sm + 3 * q * LP + t * Pad::RP;
    V v0[RL], v1[RL], v2[RL];
#pragma unroll
    for (int m = 0; m < RL; m++) {
      v0[m] = s[m];
      v1[m] = s[LP + m];
      v2[m] = s[2 * LP + m];
    }
    DftN<RL, false, V>::run(v0);
    DftN<RL, false, V>::run(v1);
    DftN<RL, false, V>::run(v2);
    const bool fx = (f0 + q) & 2, fz = (f0 + q) & 1;
    const int k0 = block_freq<PY>(t);
#pragma unroll
    for (int m = 0; m < RL; m++) {
      const int ky = k0 + m * NB;
      const bool fy = ky > N / 2;
      T2 d[6];
      load_d6(sd + (fy ? N - ky : ky) * 6, d);
      flip(d[1], fx != fy);  // xy: odd in x and y
      flip(d[2], fx != fz);  // xz
      flip(d[4], fy != fz);  // yz
      dmul(d, v0[m], v1[m], v2[m]);
    }
    DftN<RL, true, V>::run(v0);
    DftN<RL, true, V>::run(v1);
    DftN<RL, true, V>::run(v2);
#pragma unroll
    for (int m = 0; m < RL; m++) {
      s[m] = v0[m];
      s[LP + m] = v1[m];
      s[2 * LP + m] = v2[m];
    }
  }
  __syncthreads();
  pass_middles<PY, true, 1, K - 1, V, T2, false, NT>(sm, RQ * 3, tw, at);
  for (int it = threadIdx.x; it < RQ * 3 * S0; it += NT) {
    const int j = it % S0, rc = it / S0, q = rc / 3, c = rc - 3 * q;
    if (!row_on(q)) continue;
    V* dst = row_ptr(q) + c * p.by;
    const V* s = sm + rc * LP + Pad::at(j);
    V v[R];
#pragma unroll
    for (int m = 0; m < R; m++) v[m] = s[Pad::at(m * S0)];
    pass_twiddle<PY, 0, true>(v, j, tw);
    DftN<R, true, V>::run(v);
#pragma unroll
    for (int m = 0; m < NZ; m++) {
      const int y = j + m * S0;
      if (y < p.by) dst[y] = v[m];
    }
  }
}

// The three kernels of one precision and width, as the host launches them.
template <typename T, int W> struct PassKernels {
  typedef typename C2<T>::t T2;
  typedef typename PassV<T, W>::t V;
  void (*zfwd)(const T2*, V*, PassGeom, const T2*, const KrylovState*, int) = nullptr;
  void (*zinv)(T2*, const V*, PassGeom, const T2*, const KrylovState*, int) = nullptr;
  void (*rows)(V*, const T2*, PassGeom, const T2*, const KrylovState*, int) = nullptr;
  int ztc = 0, ntf = 0, nti = 0, ntr = 0, rows_per = 0;  // column tile, threads, CTAs per octant row
  size_t smem_z = 0, smem_rows = 0;
};

// Pairs of right-hand sides pay while a first butterfly of them fits the
// registers (240 = 30 x 8: z forward, z inverse and rows 118, 117 and 310 us in
// pairs, 103, 121 and 263 one by one).
template <int W, typename P> constexpr bool pass_width() { return W == 1 || P::r[0] < 30; }

template <typename T, int W, typename P> void pass_z(PassKernels<T, W>& k) {
  if constexpr (!pass_width<W, P>()) return;
  else {
    typedef ZTile<typename PassV<T, W>::t, P> Z;
    k.zfwd = k_zfwd<T, W, P>;
    k.zinv = k_zinv<T, W, P>;
    k.ztc = Z::TC;
    k.ntf = Z::NTF;
    k.nti = Z::NTI;
    k.smem_z = (size_t)P::N * Z::SEG + StageTw<P>::count() * sizeof(typename C2<T>::t);
  }
}
template <typename T, int W, typename P> void pass_y(PassKernels<T, W>& k) {
  if constexpr (!pass_width<W, P>()) return;
  else {
    typedef RTile<typename PassV<T, W>::t, P> R;
    k.rows = k_rows<T, W, P>;
    k.ntr = R::NT;
    k.rows_per = 4 / R::RQ;
    k.smem_rows = rows_smem<T, W, P>();
  }
}

}  // namespace dda
