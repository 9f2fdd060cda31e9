// farfield_kernels.cuh -- scattered far field of the dipole polarisations for
// many directions at once.
//
// FieldCalculator::calcField (DDA/CpuFieldCalculator.cpp:48-98, GPU kernel
// DDA/GpuFieldCalculatorInst.cl:27-70, launched once per direction from a
// host loop in DDA/FarFieldCalc.cpp:131-155) computes for one direction n
//   S = sum_j P_j exp(-i kd n.r_j),  E = i k^2 exp(-i k origin.n) (S - n (n.S)).
// Here a CTA takes DB directions of one right-hand side and walks the
// dipoles line by line: the y/z phase is one sincos per line and direction,
// the x phase comes from a per-CTA table, and all sums are FP64.
#pragma once

#include "fft_engine.cuh"

namespace dda {

struct FfGeom {
  int nv, nvs, by, nlines, bx;
  double kd, k;             // kd and wave number
  double ox, oy, oz;        // particle origin (metres)
};

template <typename T, int NT, int DB>
__global__ void __launch_bounds__(NT) k_farfield(const typename C2<T>::t* __restrict__ pol,
                                                 const uint32_t* __restrict__ line_off,
                                                 const uint32_t* __restrict__ dip,
                                                 const uint32_t* __restrict__ perm,
                                                 const double* __restrict__ dirs, int ndir, FfGeom g,
                                                 double2* __restrict__ out) {
  typedef typename C2<T>::t T2;
  extern __shared__ __align__(16) unsigned char ffsm[];
  double2* tx = reinterpret_cast<double2*>(ffsm);  // [DB][bx]
  __shared__ double nd[DB][3];
  __shared__ double2 red[NT / 32][DB][3];
  const int d0 = blockIdx.x * DB, b = blockIdx.y;
  const int nd_here = min(DB, ndir - d0);
  if (threadIdx.x < DB * 3) {
    const int d = threadIdx.x / 3, a = threadIdx.x % 3;
    nd[d][a] = d < nd_here ? dirs[(size_t)(d0 + d) * 3 + a] : 0.0;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < DB * g.bx; i += NT) {
    const int d = i / g.bx, x = i % g.bx;
    double s, c;
    sincos(-g.kd * nd[d][0] * (double)x, &s, &c);
    tx[i] = make_double2(c, s);
  }
  __syncthreads();
  const T2* P = pol + (size_t)b * 3 * g.nvs;
  double2 acc[DB][3];
#pragma unroll
  for (int d = 0; d < DB; d++)
#pragma unroll
    for (int c = 0; c < 3; c++) acc[d][c] = make_double2(0, 0);
  for (int L = threadIdx.x; L < g.nlines; L += NT) {
    const uint32_t j0 = line_off[L], j1 = line_off[L + 1];
    if (j0 == j1) continue;
    const int z = L / g.by, y = L - z * g.by;
    double2 ls[DB][3];
#pragma unroll
    for (int d = 0; d < DB; d++)
#pragma unroll
      for (int c = 0; c < 3; c++) ls[d][c] = make_double2(0, 0);
    for (uint32_t j = j0; j < j1; j++) {
      const int x = (int)(dip[j] & 0xffffu);
      const uint32_t jj = perm ? perm[j] : j;
      double2 p[3];
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const T2 v = P[c * g.nvs + jj];
        p[c] = make_double2(v.x, v.y);
      }
#pragma unroll
      for (int d = 0; d < DB; d++) {
        const double2 t = tx[d * g.bx + x];
#pragma unroll
        for (int c = 0; c < 3; c++) {
          ls[d][c].x += p[c].x * t.x - p[c].y * t.y;
          ls[d][c].y += p[c].x * t.y + p[c].y * t.x;
        }
      }
    }
#pragma unroll
    for (int d = 0; d < DB; d++) {
      double s, c;
      sincos(-g.kd * (nd[d][1] * y + nd[d][2] * z), &s, &c);
#pragma unroll
      for (int k = 0; k < 3; k++) {
        acc[d][k].x += ls[d][k].x * c - ls[d][k].y * s;
        acc[d][k].y += ls[d][k].x * s + ls[d][k].y * c;
      }
    }
  }
  // block reduction in a fixed order
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int d = 0; d < DB; d++)
#pragma unroll
    for (int c = 0; c < 3; c++) {
      double2 v = acc[d][c];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        v.x += __shfl_down_sync(0xffffffffu, v.x, o);
        v.y += __shfl_down_sync(0xffffffffu, v.y, o);
      }
      if (lane == 0) red[w][d][c] = v;
    }
  __syncthreads();
  if (threadIdx.x < nd_here) {
    const int d = threadIdx.x;
    double2 S[3];
    for (int c = 0; c < 3; c++) {
      S[c] = make_double2(0, 0);
      for (int ww = 0; ww < NT / 32; ww++) {
        S[c].x += red[ww][d][c].x;
        S[c].y += red[ww][d][c].y;
      }
    }
    const double* n = nd[d];
    const double2 ndS = make_double2(n[0] * S[0].x + n[1] * S[1].x + n[2] * S[2].x,
                                     n[0] * S[0].y + n[1] * S[1].y + n[2] * S[2].y);
    double s, c;
    sincos(-g.k * (g.ox * n[0] + g.oy * n[1] + g.oz * n[2]), &s, &c);
    const double k2 = g.k * g.k;
    // f = i k^2 exp(-i k origin.n)
    const double fx = -k2 * s, fy = k2 * c;
    for (int a = 0; a < 3; a++) {
      const double tx_ = S[a].x - n[a] * ndS.x, ty_ = S[a].y - n[a] * ndS.y;
      out[((size_t)(d0 + d) * gridDim.y + b) * 3 + a] = make_double2(fx * tx_ - fy * ty_, fx * ty_ + fy * tx_);
    }
  }
}

// ---- many directions: directions on the lanes -------------------------------
// The sum is a product of the dipoles' polarisations with one phase per
// (dipole, direction), 12 double-precision FMAs per dipole, direction and
// right-hand side, which bound it.  k_farfield walks a line per thread, so
// neighbouring threads read polarisations a line apart, every CTA reads all of
// them for four directions, and its warps wait for those loads.  Here a lane
// holds DL directions and their sums of NR right-hand sides: a warp stages 32
// dipoles of a line in shared memory with consecutive loads, and each lane
// reads them back as broadcasts, so one read serves 32 DL directions (DL = 2
// where NR = 1, see the host's rule).  64 x 48 x 48 ellipsoid (77 000 dipoles),
// 5 551 directions, two right-hand sides: 1.2 ms of 0.55 ms at the FMA rate,
// the shared-memory reads (11 wavefronts a dipole) taking about as long as
// the 24 FMAs.
//
// grid (ceil(ndir / (32 DL)), splits, ceil(nrhs / NR)): warp w of split s takes
// lines s 8 + w, s 8 + w + 8 splits, ...  (neighbouring lines have like
// lengths).  Partial sums go to part[split][direction][rhs][3], added in
// order by k_ff_combine.  Shared memory: x phases [bx][32 DL], then the warps'
// dipoles, reused for the warps' sums.
constexpr int kNtFf = 256;
template <int NR, int DL> __host__ __device__ constexpr size_t ff_part_smem(int bx) {
  return ((size_t)bx * 32 * DL + (kNtFf / 32) * NR * 3 * 32 * DL) * sizeof(double2) + kNtFf * sizeof(int);
}

template <typename T, int NR, int DL>
__global__ void __launch_bounds__(kNtFf, 2 / DL) k_ff_part(const typename C2<T>::t* __restrict__ pol,
                                                           const uint32_t* __restrict__ line_off,
                                                           const uint32_t* __restrict__ dip,
                                                           const uint32_t* __restrict__ perm,
                                                           const double* __restrict__ dirs, int ndir, int nrhs,
                                                           FfGeom g, double2* __restrict__ part) {
  typedef typename C2<T>::t T2;
  constexpr int NW = kNtFf / 32, ND = 32 * DL, Q = NR * 3;
  extern __shared__ __align__(16) unsigned char ffsm[];
  double2* tx = reinterpret_cast<double2*>(ffsm);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double2* all = tx + (size_t)g.bx * ND;
  double2* mine = all + w * Q * ND;
  int* xs = reinterpret_cast<int*>(all + NW * Q * ND) + w * 32;
  const int d0 = blockIdx.x * ND, r0 = blockIdx.z * NR, split = blockIdx.y, splits = gridDim.y;
  double ny[DL], nz[DL];
#pragma unroll
  for (int u = 0; u < DL; u++) {
    const double* n = dirs + (size_t)min(d0 + u * 32 + lane, ndir - 1) * 3;
    ny[u] = n[1];
    nz[u] = n[2];
    for (int x = w; x < g.bx; x += NW) {
      double s, c;
      sincos(-g.kd * n[0] * (double)x, &s, &c);
      tx[x * ND + u * 32 + lane] = make_double2(c, s);
    }
  }
  __syncthreads();
  double2 acc[DL][Q];
#pragma unroll
  for (int u = 0; u < DL; u++)
#pragma unroll
    for (int q = 0; q < Q; q++) acc[u][q] = make_double2(0, 0);
  for (int L = split * NW + w; L < g.nlines; L += NW * splits) {
    const uint32_t j0 = line_off[L], j1 = line_off[L + 1];
    if (j0 == j1) continue;
    double2 ls[DL][Q];
#pragma unroll
    for (int u = 0; u < DL; u++)
#pragma unroll
      for (int q = 0; q < Q; q++) ls[u][q] = make_double2(0, 0);
    for (uint32_t jb = j0; jb < j1; jb += 32) {
      const int cnt = min(32, (int)(j1 - jb));
      if (lane < cnt) {
        const uint32_t j = jb + lane, jj = perm ? perm[j] : j;
        xs[lane] = (int)(dip[j] & 0xffffu) * ND;
#pragma unroll
        for (int r = 0; r < NR; r++)
          if (r0 + r < nrhs) {
            const T2* P = pol + (size_t)(r0 + r) * 3 * g.nvs + jj;
#pragma unroll
            for (int c = 0; c < 3; c++) {
              const T2 v = P[(size_t)c * g.nvs];
              mine[(r * 3 + c) * 32 + lane] = make_double2(v.x, v.y);
            }
          }
      }
      __syncwarp();
#pragma unroll 2
      for (int k = 0; k < cnt; k++) {
        double2 t[DL];
#pragma unroll
        for (int u = 0; u < DL; u++) t[u] = tx[xs[k] + u * 32 + lane];
#pragma unroll
        for (int q = 0; q < Q; q++) {
          const double2 p = mine[q * 32 + k];
#pragma unroll
          for (int u = 0; u < DL; u++) {
            ls[u][q].x = fma(-p.y, t[u].y, fma(p.x, t[u].x, ls[u][q].x));
            ls[u][q].y = fma(p.y, t[u].x, fma(p.x, t[u].y, ls[u][q].y));
          }
        }
      }
      __syncwarp();
    }
    const int z = L / g.by, y = L - z * g.by;
#pragma unroll
    for (int u = 0; u < DL; u++) {
      double s, c;
      sincos(-g.kd * (ny[u] * y + nz[u] * z), &s, &c);
#pragma unroll
      for (int q = 0; q < Q; q++) {
        acc[u][q].x += ls[u][q].x * c - ls[u][q].y * s;
        acc[u][q].y += ls[u][q].x * s + ls[u][q].y * c;
      }
    }
  }
  // the CTA's sum, warps in order, through the staging area
#pragma unroll
  for (int u = 0; u < DL; u++)
#pragma unroll
    for (int q = 0; q < Q; q++) mine[q * ND + u * 32 + lane] = acc[u][q];
  __syncthreads();
  for (int i = threadIdx.x; i < Q * ND; i += kNtFf) {
    double2 t = make_double2(0, 0);
    for (int k = 0; k < NW; k++) {
      t.x += all[k * Q * ND + i].x;
      t.y += all[k * Q * ND + i].y;
    }
    const int q = i / ND, dd = d0 + i % ND, r = r0 + q / 3;
    if (dd < ndir && r < nrhs) part[(((size_t)split * ndir + dd) * nrhs + r) * 3 + q % 3] = t;
  }
}

// E of one (direction, right-hand side) per thread from its partial sums.
__global__ void k_ff_combine(const double2* __restrict__ part, int splits, const double* __restrict__ dirs, int ndir,
                             int nrhs, FfGeom g, double2* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ndir * nrhs) return;
  const double* n = dirs + (size_t)(i / nrhs) * 3;
  double2 S[3];
  for (int c = 0; c < 3; c++) S[c] = make_double2(0, 0);
  for (int k = 0; k < splits; k++)
    for (int c = 0; c < 3; c++) {
      const double2 p = part[((size_t)k * ndir * nrhs + i) * 3 + c];
      S[c].x += p.x;
      S[c].y += p.y;
    }
  const double2 ndS = make_double2(n[0] * S[0].x + n[1] * S[1].x + n[2] * S[2].x,
                                   n[0] * S[0].y + n[1] * S[1].y + n[2] * S[2].y);
  double s, c;
  sincos(-g.k * (g.ox * n[0] + g.oy * n[1] + g.oz * n[2]), &s, &c);
  const double k2 = g.k * g.k, fx = -k2 * s, fy = k2 * c;  // f = i k^2 exp(-i k origin.n)
  for (int a = 0; a < 3; a++) {
    const double tx = S[a].x - n[a] * ndS.x, ty = S[a].y - n[a] * ndS.y;
    out[(size_t)i * 3 + a] = make_double2(fx * tx - fy * ty, fx * ty + fy * tx);
  }
}

}  // namespace dda
