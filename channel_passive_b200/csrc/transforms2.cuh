// transforms2.cuh - the four-step transform kernels, shared by transforms2.cu (the tuned lengths) and
// transforms3.cu (the others).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include "fft2.cuh"
#include "kmm_internal.h"
#include "stats.cuh"
#include "tma.cuh"

namespace kmm {

namespace {

template <typename C> __device__ __forceinline__ C ld_as(const double2 *p) {
  const double2 v = *p;
  return cmake<C>(v.x, v.y);
}
template <typename R> __device__ __forceinline__ const typename Cpx<R>::T *tw_of(const FftPlan &pl);
template <> __device__ __forceinline__ const double2 *tw_of<double>(const FftPlan &pl) { return pl.tw64; }
template <> __device__ __forceinline__ const float2 *tw_of<float>(const FftPlan &pl) { return pl.tw32; }

// Threads of a z-transform block: one per (line, step-1 or step-2 work item).
template <int N1, int N2, int KB>
constexpr int z_threads() {
  return KB * (N1 > N2 ? N1 : N2);
}

// The z position of padded index p (3/2 rule of ppdfftw_dft_z_inverse, module_ppdfftw.f90:846-854):
// kz index for p < nz/2 and p > nz, -1 for the zero band nz/2..nz.
__device__ __forceinline__ int zpad_src(int p, int nh) { return p < nh ? p : (p > 2 * nh ? p - nh : -1); }

// ---- TMA staging of the z-transform input tiles (cp.async.bulk.tensor, no multicast) -------
// A block's input tile (its KB kx columns of all rows of one (field, y) plane) is copied into
// shared memory as 3-D tensor boxes of (2 KB scalars, tile_rows(n) rows, 1 plane); the copies
// complete on an mbarrier whose wait has an iteration limit.
// Rows of one TMA box over n rows: n split into ceil(n / 256) equal boxes (0 if they are not equal).
__host__ __device__ constexpr int tile_rows(int n) {
  const int nb = (n + 255) / 256;
  return n % nb == 0 ? n / nb : 0;
}

__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, int x, int y, int z, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}

// Copies a block's tile (KB columns x n rows of element E) into `base`, in tile_rows(n)-row boxes,
// and waits for it.  Thread 0 arms the barrier and issues the copies; every thread waits (the
// completed phase makes the bytes visible to it).  Returns false, for the whole block, if the
// wait gave up: the error flag is set and the block should leave.
template <typename E, int KB>
__device__ __forceinline__ bool tma_tile(unsigned char *base, const CUtensorMap *map, int n, int x, int plane,
                                         uint64_t *bar, int *err) {
  if (threadIdx.x == 0) mbar_init(bar, 1);
  __syncthreads();
  if (threadIdx.x == 0) {
    const int rows = tile_rows(n);
    mbar_expect_tx(bar, (unsigned)(KB * n * sizeof(E)));
    for (int r0 = 0; r0 < n; r0 += rows) tma_load_3d(base + (size_t)r0 * KB * sizeof(E), map, x, r0, plane, bar);
  }
  const bool ok = mbar_wait_bounded(bar);
  if (__syncthreads_or(!ok)) {
    // the copy did not complete: flag it and give it one more bounded wait before the block leaves
    if (threadIdx.x == 0) atomicCAS(err, 0, KMM_ERR_TIMEOUT);
    mbar_wait_bounded(bar);
    return false;
  }
  return true;
}

// Dynamic shared memory of a z kernel with TMA: the larger of the tile and the FFT lines (the lines
// overlay the tile once every thread has taken its inputs), plus 128 bytes so that the tile can
// start on a 128-byte shared address.
template <typename R, int N1, int N2, int KB, typename E>
constexpr size_t z_smem_tma(int n) {
  const size_t tile = (size_t)KB * n * sizeof(E);
  const size_t lines = (size_t)KB * ip_lda<N1, N2>() * sizeof(typename Cpx<R>::T);
  return (tile > lines ? tile : lines) + 128;
}

// y_to_x: grid (ceil(nxh/KB), ny, nfield).  Thread (l, n1) of step 1 reads its N2 points
// x[n1 + N1*n2] of kx line l straight from the Y-pencil (16 consecutive kx per row: one coalesced
// run) or, with TMA, from the block's tile in shared memory, transforms them in registers and
// leaves them in shared memory; thread (l, k2) of step 2 finishes the line and writes
// X[k2 + N2*k1] straight into the X-pencil slab.
template <typename R, int N1, int N2, int KB, bool TMA = false>
__global__ void __launch_bounds__(z_threads<N1, N2, KB>()) k_zinv2(const double2 *__restrict__ src,
                                                                  typename Cpx<R>::T *__restrict__ dst,
                                                                  FftPlan pl, int nz, int nxh, int64_t ns,
                                                                  int64_t nm, const __grid_constant__ CUtensorMap tmap,
                                                                  int ny, int *err) {
  using C = typename Cpx<R>::T;
  constexpr int N = N1 * N2, LD = ip_lda<N1, N2>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  // with TMA the tile (and the lines over it) starts on the next 128-byte shared address
  unsigned char *base = TMA ? smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u) : smem_raw;
  C *a = reinterpret_cast<C *>(base);
  const int nh = nz / 2;
  const int kx0 = blockIdx.x * KB, y = blockIdx.y, f = blockIdx.z;
  const int l = threadIdx.x % KB, item = threadIdx.x / KB;
  const bool live = kx0 + l < nxh;
  const C *tw = tw_of<R>(pl);
  C v[N2];
  if constexpr (TMA) {
    __shared__ __align__(8) uint64_t bar;
    if (!tma_tile<double2, KB>(base, &tmap, nz, 2 * kx0, f * ny + y, &bar, err)) return;
    const double2 *tile = reinterpret_cast<const double2 *>(base);
    if (item < N1) {
      const int n1 = item;
#pragma unroll
      for (int n2 = 0; n2 < N2; ++n2) {
        const int kzi = zpad_src(n1 + N1 * n2, nh);
        v[n2] = (live && kzi >= 0) ? ld_as<C>(tile + kzi * KB + l) : cmake<C>(0.0, 0.0);
      }
    }
    __syncthreads();  // the FFT lines overlay the tile
  } else {
    if (item < N1) {
      const int n1 = item;
      const double2 *sp = src + f * ns + (int64_t)y * nz * nxh + kx0 + l;
#pragma unroll
      for (int n2 = 0; n2 < N2; ++n2) {
        const int kzi = zpad_src(n1 + N1 * n2, nh);
        v[n2] = (live && kzi >= 0) ? ld_as<C>(sp + (int64_t)kzi * nxh) : cmake<C>(0.0, 0.0);
      }
    }
  }
  if (item < N1) {
    const int n1 = item;
    reg_dft<C, N2>(v, +1);
    C *yl = a + l * LD;
    yl[n1] = v[0];
#pragma unroll
    for (int k2 = 1; k2 < N2; ++k2) {
      C w = tw[n1 * k2];
      w.y = -w.y;
      yl[n1 + (N1 + 1) * k2] = n1 > 0 ? cmul(v[k2], w) : v[k2];
    }
  }
  __syncthreads();
  if (item < N2 && live) {
    const int k2 = item;
    const C *yl = a + l * LD;
    C v[N1];
#pragma unroll
    for (int n1 = 0; n1 < N1; ++n1) v[n1] = yl[n1 + (N1 + 1) * k2];
    reg_dft<C, N1>(v, +1);
    C *dp = dst + f * nm + (int64_t)y * N * nxh + kx0 + l;
#pragma unroll
    for (int k1 = 0; k1 < N1; ++k1) dp[(int64_t)(k2 + N2 * k1) * nxh] = v[k1];
  }
}

// x_to_y: grid (ceil(nxh/KB), ny, nfield).  The mirror of k_zinv2: step 1 reads the X-pencil
// slab, step 2 writes the kept frequencies (truncation of ppdfftw_dft_z_forward,
// module_ppdfftw.f90:811-817) with the kz Nyquist row zeroed and the rescale folded in.
// With TMA, step 1 takes its points from the block's tile of the slab (KB kx columns of the N
// rows of one (field, y) plane), which the FFT lines then overlay.
template <typename R, int N1, int N2, int KB, typename D, bool TMA = false>
__global__ void __launch_bounds__(z_threads<N1, N2, KB>()) k_zfwd2(const typename Cpx<R>::T *__restrict__ src,
                                                                  D *__restrict__ dst, FftPlan pl, int nz, int nxh,
                                                                  int64_t ns, int64_t nm, double scale,
                                                                  const __grid_constant__ CUtensorMap tmap, int ny,
                                                                  int *err) {
  using C = typename Cpx<R>::T;
  constexpr int N = N1 * N2, LD = ip_lda<N1, N2>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned char *base = TMA ? smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u) : smem_raw;
  C *a = reinterpret_cast<C *>(base);
  const int nh = nz / 2;
  const int kx0 = blockIdx.x * KB, y = blockIdx.y, f = blockIdx.z;
  const int l = threadIdx.x % KB, item = threadIdx.x / KB;
  const bool live = kx0 + l < nxh;
  const C *tw = tw_of<R>(pl);
  C v[N2];
  if constexpr (TMA) {
    __shared__ __align__(8) uint64_t bar;
    if (!tma_tile<C, KB>(base, &tmap, N, 2 * kx0, f * ny + y, &bar, err)) return;
    const C *tile = reinterpret_cast<const C *>(base);
    if (item < N1) {
      const int n1 = item;
#pragma unroll
      for (int n2 = 0; n2 < N2; ++n2) v[n2] = live ? tile[(n1 + N1 * n2) * KB + l] : cmake<C>(0.0, 0.0);
    }
    __syncthreads();  // the FFT lines overlay the tile
  } else {
    if (item < N1) {
      const int n1 = item;
      const C *sp = src + f * nm + (int64_t)y * N * nxh + kx0 + l;
#pragma unroll
      for (int n2 = 0; n2 < N2; ++n2) v[n2] = live ? sp[(int64_t)(n1 + N1 * n2) * nxh] : cmake<C>(0.0, 0.0);
    }
  }
  if (item < N1) {
    const int n1 = item;
    reg_dft<C, N2>(v, -1);
    C *yl = a + l * LD;
    yl[n1] = v[0];
#pragma unroll
    for (int k2 = 1; k2 < N2; ++k2) yl[n1 + (N1 + 1) * k2] = n1 > 0 ? cmul(v[k2], tw[n1 * k2]) : v[k2];
  }
  __syncthreads();
  if (item < N2 && live) {
    const int k2 = item;
    const C *yl = a + l * LD;
    C v[N1];
#pragma unroll
    for (int n1 = 0; n1 < N1; ++n1) v[n1] = yl[n1 + (N1 + 1) * k2];
    reg_dft<C, N1>(v, -1);
    D *dp = dst + f * ns + (int64_t)y * nz * nxh + kx0 + l;
#pragma unroll
    for (int k1 = 0; k1 < N1; ++k1) {
      const int k = k2 + N2 * k1;
      int kzi = -1;
      D out;
      if (k < nh || k > 2 * nh) {
        kzi = k < nh ? k : k - nh;
        out.x = (decltype(out.x))(scale * (double)v[k1].x);
        out.y = (decltype(out.y))(scale * (double)v[k1].y);
      } else if (k == nh) {  // the kz Nyquist row is zeroed (module_ppdfftw.f90:811-817)
        kzi = nh;
        out.x = 0;
        out.y = 0;
      }
      if (kzi >= 0) dp[(int64_t)kzi * nxh] = out;
    }
  }
}

struct X2Args {
  int ny, nz32, nxh;
  float rnxh;  // 1 / nxh: the loops below split w into (w / nxh, w % nxh) without an integer divide
  int64_t nm;
  double dxr, dzr;
  const double *dyr;
  int substep;
  DevScalars *dsc;
  double *mom;  // STAT only, may be null: per-block moment sums [ny][gridDim.x][kNumMoments]
};

// dft_x_realspace: grid (ceil(nz32/ZB), ny), NT threads; MID slots 0..3 = u, v, w, theta in,
// slots 0..7 = f1, f2, f3, f4, f5, f7, f8, f9 out (a block owns its rows).
// STAT: the statistics-step products for the pressure instead (f1..f6 with f6 = v v,
// dft_x_realspace.f90:192-199): packed lines (f1, f2), (f3, f4), (f5, f6); no CFL, and only
// slots 0..5 are written.  With a_.mom set, each block also writes the sums over its physical
// points of the moments of dft_x_realspace.f90:128-155 (moment_terms), in FP64.
#ifndef KMM_X576_MINB
#define KMM_X576_MINB 5
#endif
// Resident blocks asked of the compiler: at N = 576 the FP32 step pass otherwise takes 140
// registers a thread, 3 blocks (12 warps) an SM.  5 blocks (96 registers, a 200-byte spill) took
// the pass from 2.35 to 2.01 ms on the 384x257x384 grid (4 blocks, no spill: 2.04 ms).  The
// statistics variant keeps the default: a cap spills more there.
// At N = 288 (16 x 18) the FP32 step pass took 80 registers, 6 blocks an SM; 8 blocks (64
// registers, a 56-byte spill) took it from 0.2345 to 0.2155 ms on the 192x129x192 grid
// (7 blocks: 0.2167 ms).
#ifndef KMM_X288_MINB
#define KMM_X288_MINB 8
#endif
// The FP64 step pass at N = 288 took 152 registers with 64 threads, 6 blocks (12 warps) an SM;
// 8 blocks (128 registers, a 64-byte spill) took it from 0.3887 to 0.3712 ms.
#ifndef KMM_X288_MINB_FP64
#define KMM_X288_MINB_FP64 8
#endif
template <typename R, int N, bool STAT, int NS = 1, int V = 0> constexpr int x_min_blocks() {
  if (STAT || V != 0) return 1;  // the caps below were measured for the default shape
  // two scalars, FP32 at N = 576: 210 registers uncapped (2 blocks an SM); 3 blocks fit the
  // shared memory of the six packed lines per row
  if (NS != 1) return (sizeof(R) == 4 && N >= 576) ? 3 : 1;
  if (sizeof(R) != 4) return N == 288 ? KMM_X288_MINB_FP64 : 1;
  return N >= 576 ? KMM_X576_MINB : N == 288 ? KMM_X288_MINB : 1;
}

// NS = 2: a second passive scalar theta2 in MID slot 4; its products u theta2, v theta2, w theta2
// go to slots 8, 9, 10, formed like f7..f9 (a third packed input line (theta2, 0) and two packed
// output lines (u theta2, v theta2), (w theta2, 0)).
template <typename R, int N1, int N2, int ZB, int NT, bool STAT = false, int NS = 1, int V = 0>
__global__ void __launch_bounds__(NT, (x_min_blocks<R, N1 * N2, STAT, NS, V>())) k_xphys2(typename Cpx<R>::T *__restrict__ mid, FftPlan pl, X2Args a_) {
  using C = typename Cpx<R>::T;
  constexpr int N = N1 * N2, LD = ip_lda<N1, N2>();
  constexpr int NIN = 1 + NS, NOUT = 2 + 2 * NS;  // packed input and output lines per row
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C *a = reinterpret_cast<C *>(smem_raw);  // NOUT*ZB lines: (u,v) ZB, (w,theta) ZB, [(theta2,0) ZB,] then outputs
  const int nxh = a_.nxh;
  const int z0 = blockIdx.x * ZB, y = blockIdx.y;
  const int64_t row0 = ((int64_t)y * a_.nz32 + z0) * nxh;
  for (int w = threadIdx.x; w < NIN * ZB * N; w += NT) {
    const int L = w / N, p = w - L * N;
    a[L * LD + p] = cmake<C>(0.0, 0.0);
  }
  __syncthreads();
  // Z_k = X1_k + i X2_k and its Hermitian mirror at N - k; DC imaginary parts dropped (c2r)
  for (int w = threadIdx.x; w < NIN * ZB * nxh; w += NT) {
    // exact: (w + 0.5) / nxh stays at least 0.5 / nxh away from an integer, far above float rounding
    const int t = (int)(((float)w + 0.5f) * a_.rnxh), k = w - t * nxh, l = t % ZB, bsel = t / ZB;
    if (z0 + l >= a_.nz32) continue;
    const int64_t off = row0 + (int64_t)l * nxh + k;
    const int fa = bsel == 0 ? 0 : bsel == 1 ? 2 : 4, fb = bsel == 0 ? 1 : 3;
    const C x1 = mid[fa * a_.nm + off];
    const C x2 = bsel < 2 ? mid[fb * a_.nm + off] : cmake<C>(0.0, 0.0);
    C *line = a + (bsel * ZB + l) * LD;
    if (k == 0) {
      line[0] = cmake<C>(x1.x, x2.x);
    } else {
      C zk, zm;
      zk.x = x1.x - x2.y; zk.y = x1.y + x2.x;
      zm.x = x1.x + x2.y; zm.y = x2.x - x1.y;
      line[k] = zk;
      line[N - k] = zm;
    }
  }
  __syncthreads();
  fft4_ip<R, N1, N2, NIN * ZB, NT>(a, LD, tw_of<R>(pl), +1);
  const double dyr = a_.dyr[y];
  double vmax = 0.0;
  int bad = 0;
  double ms[STAT ? kNumMoments : 1] = {};
  for (int w = threadIdx.x; w < ZB * N; w += NT) {
    const int l = w / N, p = w - l * N;
    const C uv = a[l * LD + p], wt = a[(ZB + l) * LD + p];
    const R u = uv.x, v = uv.y, ww = wt.x, t = wt.y;
    R t2 = 0;
    if constexpr (NS == 2) t2 = a[(2 * ZB + l) * LD + p].x;
    if constexpr (STAT) {
      if (a_.mom && z0 + l < a_.nz32) moment_terms(ms, (double)u, (double)v, (double)ww);
    }
    const R bv2 = v * v;
    C f12, f34, f57, f89;
    f12.x = u * u - bv2; f12.y = u * v;
    f34.x = ww * ww - bv2; f34.y = v * ww;
    if constexpr (STAT) {
      f57.x = u * ww; f57.y = bv2;
      f89.x = 0; f89.y = 0;
    } else {
      f57.x = u * ww; f57.y = u * t;
      f89.x = v * t; f89.y = ww * t;
    }
    a[l * LD + p] = f12;
    a[(ZB + l) * LD + p] = f34;
    a[(2 * ZB + l) * LD + p] = f57;
    a[(3 * ZB + l) * LD + p] = f89;
    if constexpr (NS == 2) {
      C g12, g3;
      g12.x = u * t2; g12.y = v * t2;
      g3.x = ww * t2; g3.y = 0;
      a[(4 * ZB + l) * LD + p] = g12;
      a[(5 * ZB + l) * LD + p] = g3;
    }
    if (!STAT && a_.substep == 1 && z0 + l < a_.nz32) {
      const double vel = (fabs((double)u) * a_.dxr) + (fabs((double)v) * dyr) + (fabs((double)ww) * a_.dzr);
      if (!isfinite(vel)) bad = 1;
      else vmax = fmax(vmax, vel);
    }
  }
  __syncthreads();
  fft4_ip<R, N1, N2, NOUT * ZB, NT>(a, LD, tw_of<R>(pl), -1);
  for (int w = threadIdx.x; w < (STAT ? 3 : NOUT) * ZB * nxh; w += NT) {
    // exact: (w + 0.5) / nxh stays at least 0.5 / nxh away from an integer, far above float rounding
    const int t = (int)(((float)w + 0.5f) * a_.rnxh), k = w - t * nxh, l = t % ZB, bsel = t / ZB;
    if (z0 + l >= a_.nz32) continue;
    const C *line = a + (bsel * ZB + l) * LD;
    const C zk = line[k], zm = line[k == 0 ? 0 : N - k];
    C A, B;
    A.x = (R)0.5 * (zk.x + zm.x); A.y = (R)0.5 * (zk.y - zm.y);
    B.x = (R)0.5 * (zk.y + zm.y); B.y = (R)0.5 * (zm.x - zk.x);
    const int64_t off = row0 + (int64_t)l * nxh + k;
    mid[(2 * bsel) * a_.nm + off] = A;
    if (2 * bsel + 1 < 11) mid[(2 * bsel + 1) * a_.nm + off] = B;  // slot 11 would be the zero partner
  }
  if constexpr (STAT) {
    if (a_.mom) {
      // fixed-order block sum: lanes by shuffles, then warps in order
      __shared__ double mred[NT / 32][kNumMoments];
#pragma unroll
      for (int i = 0; i < kNumMoments; ++i) {
        double x = ms[i];
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if ((threadIdx.x & 31) == 0) mred[threadIdx.x >> 5][i] = x;
      }
      __syncthreads();
      if (threadIdx.x < kNumMoments) {
        double x = 0.0;
        for (int j = 0; j < NT / 32; ++j) x += mred[j][threadIdx.x];
        a_.mom[((int64_t)y * gridDim.x + blockIdx.x) * kNumMoments + threadIdx.x] = x;
      }
    }
  }
  if (!STAT && a_.substep == 1) {
    __shared__ double red[NT / 32];
    __shared__ int redbad;
    if (threadIdx.x == 0) redbad = 0;
    __syncthreads();
    if (bad) atomicOr(&redbad, 1);
    for (int o = 16; o > 0; o >>= 1) vmax = fmax(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = vmax;
    __syncthreads();
    if (threadIdx.x == 0) {
      double m = 0.0;
      for (int i = 0; i < NT / 32; ++i) m = fmax(m, red[i]);
      atomicMax(&a_.dsc->velmax_bits, (unsigned long long)__double_as_longlong(m));
      if (redbad) atomicOr(&a_.dsc->nonfinite, 1);
    }
  }
}

template <typename K> void set_smem(K kern, int optin) {
  cudaFuncAttributes fa;
  if (cudaFuncGetAttributes(&fa, kern) != cudaSuccess) return;
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes);
}

// Lines per block (KB: z transforms, one thread per line and work item) and rows per block and
// threads (ZB, ZT: x pass), tuned at N = 288 on B200: a line needs (N1+1)*N2 | 1 complex values
// of shared memory, so these choices keep 39 KB or less per block.
template <typename R> struct TCfg;
template <> struct TCfg<float> {
  static constexpr int KB = 16, ZB = 2, ZT = 128;
};
template <> struct TCfg<double> {
  static constexpr int KB = 8, ZB = 1, ZT = 64;
};

template <typename R, int N1, int N2, int KB = TCfg<R>::KB>
constexpr size_t z_smem() {
  return sizeof(typename Cpx<R>::T) * (size_t)KB * ip_lda<N1, N2>();
}
template <typename R, int N1, int N2, int NS = 1, int ZB = TCfg<R>::ZB>
constexpr size_t x_smem() {
  return sizeof(typename Cpx<R>::T) * (size_t)(2 + 2 * NS) * ZB * ip_lda<N1, N2>();
}

[[maybe_unused]] cudaError_t fill_regtw() {
  double2 h[kRegTwTotal];
  int off = 0;
  for (int i = 0; i < kNumRegSizes; ++i) {
    const int M = kRegSizes[i];
    for (int t = 0; t < M; ++t) {
      const long double ang = -2.0L * 3.141592653589793238462643383279502884L * (long double)t / (long double)M;
      h[off + t] = make_double2((double)cosl(ang), (double)sinl(ang));
    }
    off += M;
  }
  cudaError_t e = cudaMemcpyToSymbol(c_regtw, h, sizeof(h));
  if (e != cudaSuccess) return e;
  float2 h32[kRegTwTotal];
  for (int i = 0; i < kRegTwTotal; ++i) h32[i] = make_float2((float)h[i].x, (float)h[i].y);
  return cudaMemcpyToSymbol(c_regtw32, h32, sizeof(h32));
}

X2Args x2_args(const Handle &h, int substep) {
  X2Args a;
  a.ny = h.ny;
  a.nz32 = h.nz32;
  a.nxh = h.nxh;
  a.rnxh = 1.0f / (float)h.nxh;
  a.nm = h.nm;
  a.dxr = h.dxr;
  a.dzr = h.dzr;
  a.dyr = h.dops + ops_offsets(h.bw, h.ny).dyr;
  a.substep = substep;
  a.dsc = h.dsc;
  a.mom = nullptr;
  return a;
}

}  // namespace

}  // namespace kmm
