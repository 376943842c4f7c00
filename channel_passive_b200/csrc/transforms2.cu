// transforms2.cu - the substep's transforms with compile-time four-step FFTs (fft2.cuh).
//
// Same contracts as transforms.cu (k_zinv / k_xphys / k_zfwd: y_to_x, dft_x_realspace and
// x_to_y with rescale_data folded in) for the line lengths N = N1 * N2 listed in with_shape;
// the launchers fall back to the generic kernels of transforms.cu for other lengths.  Lines
// are line-major in shared memory with the odd leading dimension (N1+1)*N2 | 1 and are
// transformed in place (fft4_ip), natural order in and out, so the 3/2 padding and truncation
// read and write plain positions k and N - k.
#include <cuda.h>
#include <cuda_runtime.h>

#include "transforms2.cuh"

namespace kmm {

namespace {

// Transpose of the x pass at a base state (the discrete adjoint; FP64), one block per x-line
// row (z, y).  With <a, b> = Re sum conj(a) b over the kept kx coefficients and the plain sum
// over physical points, the pass's three parts transpose as
//   r2c + truncate  ->  lambda_phys(x) = Re sum_{k < nxh} lambda_k e^{+ikx}: a c2r of
//                       b_0 = lambda_0, b_k = lambda_k / 2 (the same packed c2r as the forward);
//   products        ->  their linearisation at the base u, v, w, theta (a c2r of base_mid);
//   pad + c2r       ->  an r2c with weight 1 at kx = 0 (its imaginary part dropped) and 2 above.
// base_mid slots 0..3 = u, v, w, theta of the base state (x-spectral, z-physical); lmid slots
// 0..7 = lambda of f1..f5, f7..f9 on entry, multiplied by `scale` (the rescale of x_to_y), and
// lambda of u, v, w, theta in slots 0..3 on exit.
template <int N1, int N2>
__global__ void __launch_bounds__(128) k_xadj2(const double2 *__restrict__ base_mid, double2 *__restrict__ lmid,
                                              FftPlan pl, int nz32, int nxh, float rnxh, int64_t nm, double scale) {
  using C = double2;
  constexpr int N = N1 * N2, LD = ip_lda<N1, N2>(), NT = 128;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C *a = reinterpret_cast<C *>(smem_raw);  // 6 lines: base (u,v) (w,t); lambda (f1,f2) (f3,f4) (f5,f7) (f8,f9)
  const int z = blockIdx.x, y = blockIdx.y;
  const int64_t row0 = ((int64_t)y * nz32 + z) * nxh;
  for (int w = threadIdx.x; w < 6 * N; w += NT) a[(w / N) * LD + (w % N)] = make_double2(0.0, 0.0);
  __syncthreads();
  for (int w = threadIdx.x; w < 6 * nxh; w += NT) {
    const int t = (int)(((float)w + 0.5f) * rnxh), k = w - t * nxh;  // line t = 0..5, exact split
    C x1, x2;
    if (t < 2) {
      x1 = base_mid[(2 * t) * nm + row0 + k];
      x2 = base_mid[(2 * t + 1) * nm + row0 + k];
    } else {
      const double f = (k == 0 ? 1.0 : 0.5) * scale;
      const C l1 = lmid[(2 * (t - 2)) * nm + row0 + k], l2 = lmid[(2 * (t - 2) + 1) * nm + row0 + k];
      x1 = make_double2(f * l1.x, f * l1.y);
      x2 = make_double2(f * l2.x, f * l2.y);
    }
    C *line = a + t * LD;
    if (k == 0) {
      line[0] = make_double2(x1.x, x2.x);
    } else {
      line[k] = make_double2(x1.x - x2.y, x1.y + x2.x);
      line[N - k] = make_double2(x1.x + x2.y, x2.x - x1.y);
    }
  }
  __syncthreads();
  fft4_ip<double, N1, N2, 6, NT>(a, LD, tw_of<double>(pl), +1);
  for (int p = threadIdx.x; p < N; p += NT) {
    const C uv = a[p], wt = a[LD + p];
    const double u = uv.x, v = uv.y, w = wt.x, t = wt.y;
    const C l12 = a[2 * LD + p], l34 = a[3 * LD + p], l57 = a[4 * LD + p], l89 = a[5 * LD + p];
    // f1 = uu - vv, f2 = uv, f3 = ww - vv, f4 = vw, f5 = uw, f7 = u t, f8 = v t, f9 = w t
    const double lu = 2.0 * u * l12.x + v * l12.y + w * l57.x + t * l57.y;
    const double lv = -2.0 * v * l12.x + u * l12.y - 2.0 * v * l34.x + w * l34.y + t * l89.x;
    const double lw = 2.0 * w * l34.x + v * l34.y + u * l57.x + t * l89.y;
    const double lt = u * l57.y + v * l89.x + w * l89.y;
    a[2 * LD + p] = make_double2(lu, lv);
    a[3 * LD + p] = make_double2(lw, lt);
  }
  __syncthreads();
  fft4_ip<double, N1, N2, 2, NT>(a + 2 * LD, LD, tw_of<double>(pl), -1);
  for (int w = threadIdx.x; w < 2 * nxh; w += NT) {
    const int t = (int)(((float)w + 0.5f) * rnxh), k = w - t * nxh;
    const C *line = a + (2 + t) * LD;
    const C zk = line[k], zm = line[k == 0 ? 0 : N - k];
    C A = make_double2(0.5 * (zk.x + zm.x), 0.5 * (zk.y - zm.y));
    C B = make_double2(0.5 * (zk.y + zm.y), 0.5 * (zm.x - zk.x));
    if (k == 0) {
      A.y = 0.0;
      B.y = 0.0;
    } else {
      A = make_double2(2.0 * A.x, 2.0 * A.y);
      B = make_double2(2.0 * B.x, 2.0 * B.y);
    }
    lmid[(2 * t) * nm + row0 + k] = A;
    lmid[(2 * t + 1) * nm + row0 + k] = B;
  }
}

// ---- dispatch over the supported lengths ------------------------------------------------
template <typename F> bool with_shape(int N, F &&f) {
  switch (N) {
    case 12: f.template operator()<3, 4>(); return true;
    case 24: f.template operator()<4, 6>(); return true;
    case 36: f.template operator()<6, 6>(); return true;
    case 48: f.template operator()<6, 8>(); return true;
    case 72: f.template operator()<8, 9>(); return true;
    case 96: f.template operator()<8, 12>(); return true;
    case 144: f.template operator()<12, 12>(); return true;
    case 192: f.template operator()<12, 16>(); return true;
    case 288: f.template operator()<16, 18>(); return true;
    case 384: f.template operator()<16, 24>(); return true;
    case 576: f.template operator()<24, 24>(); return true;
    default: return false;
  }
}

// Tile-shape variants the autotuner (kmm_autotune) times on the handle's grid; variant 0 is the
// hand-tuned TCfg.  The others are built for lengths of kMinTunedLength points and more only
// (shorter lines fall back to variant 0 at compile time).
constexpr int kMinTunedLength = 96;
template <typename R, int V> struct ZVar;  // z transforms: lines per block
template <> struct ZVar<float, 0> { static constexpr int KB = TCfg<float>::KB; };
template <> struct ZVar<float, 1> { static constexpr int KB = 8; };
template <> struct ZVar<float, 2> { static constexpr int KB = 32; };
template <> struct ZVar<double, 0> { static constexpr int KB = TCfg<double>::KB; };
template <> struct ZVar<double, 1> { static constexpr int KB = 4; };
template <> struct ZVar<double, 2> { static constexpr int KB = 16; };
template <typename R, int V> struct XVar;  // x pass: rows per block and threads
template <> struct XVar<float, 0> { static constexpr int ZB = TCfg<float>::ZB, ZT = TCfg<float>::ZT; };
template <> struct XVar<float, 1> { static constexpr int ZB = 1, ZT = 128; };
template <> struct XVar<float, 2> { static constexpr int ZB = 4, ZT = 256; };
template <> struct XVar<double, 0> { static constexpr int ZB = TCfg<double>::ZB, ZT = TCfg<double>::ZT; };
template <> struct XVar<double, 1> { static constexpr int ZB = 1, ZT = 128; };
template <> struct XVar<double, 2> { static constexpr int ZB = 2, ZT = 128; };
template <int N, int V> constexpr int tuned_variant() { return N < kMinTunedLength ? 0 : V; }

// Runs f.template operator()<V>() for the runtime variant v (0..2).
template <typename F> void with_variant(int v, F &&f) {
  switch (v) {
    case 1: f.template operator()<1>(); break;
    case 2: f.template operator()<2>(); break;
    default: f.template operator()<0>(); break;
  }
}

}  // namespace

bool fft4_supported(int N) {
  return with_shape(N, [&]<int A, int B>() {});
}

cudaError_t prepare_transforms2() {
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  const cudaError_t e = fill_regtw();
  if (e != cudaSuccess) return e;
  for (int N : {12, 24, 36, 48, 72, 96, 144, 192, 288, 384, 576}) {
    with_shape(N, [&]<int N1, int N2>() {
      using D = TCfg<double>;
      set_smem(k_xphys2<double, N1, N2, D::ZB, D::ZT, true>, optin);
      set_smem(k_xadj2<N1, N2>, optin);
      for (int v = 0; v < 3; ++v)
        with_variant(v, [&]<int V>() {
          constexpr int VV = tuned_variant<N1 * N2, V>();
          using ZF = ZVar<float, VV>;
          using ZD = ZVar<double, VV>;
          using XF = XVar<float, VV>;
          using XD = XVar<double, VV>;
          set_smem(k_zinv2<double, N1, N2, ZD::KB>, optin);
          set_smem(k_zinv2<float, N1, N2, ZF::KB>, optin);
          set_smem(k_zfwd2<double, N1, N2, ZD::KB, double2>, optin);
          set_smem(k_zfwd2<float, N1, N2, ZF::KB, float2>, optin);
          set_smem(k_zfwd2<float, N1, N2, ZF::KB, double2>, optin);
          set_smem(k_zinv2<double, N1, N2, ZD::KB, true>, optin);
          set_smem(k_zinv2<float, N1, N2, ZF::KB, true>, optin);
          set_smem(k_zfwd2<double, N1, N2, ZD::KB, double2, true>, optin);
          set_smem(k_zfwd2<float, N1, N2, ZF::KB, float2, true>, optin);
          set_smem(k_zfwd2<float, N1, N2, ZF::KB, double2, true>, optin);
          set_smem(k_xphys2<double, N1, N2, XD::ZB, XD::ZT, false, 1, VV>, optin);
          set_smem(k_xphys2<float, N1, N2, XF::ZB, XF::ZT, false, 1, VV>, optin);
          set_smem(k_xphys2<double, N1, N2, XD::ZB, XD::ZT, false, 2, VV>, optin);
          set_smem(k_xphys2<float, N1, N2, XF::ZB, XF::ZT, false, 2, VV>, optin);
        });
    });
  }
  return cudaSuccess;
}

// The driver's tensor-map encoder (cuTensorMapEncodeTiled), fetched once through the runtime.
using EncodeTiledFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                   const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled() {
  static const EncodeTiledFn fn = [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return (EncodeTiledFn) nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}

int opt_in_smem() {
  int dev = 0, optin = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
    return 0;
  return optin;
}

// The tile map of a z kernel's input: `base` holds nfield planes per y of n rows x nxh complex
// elements of es-byte scalars (a (2 nxh, n, nfield ny) tensor of scalars); a box is KB complex
// columns by tile_rows(n) rows of one plane.  The rules of a tiled map, checked here: base and
// strides (2 nxh es, 2 nxh es n) multiples of 16 bytes, box extents <= 256, inner box 2 KB es
// bytes a multiple of 16, every copy's x coordinate 2 kx0 scalars (kx0 a multiple of KB) a
// multiple of 16 bytes, and every box's shared destination (r0 KB 2 es bytes past a 128-byte
// aligned tile) on a 128-byte boundary.  False where the grid or the encoder does not allow it;
// the caller then loads per thread.
bool z_tile_map(const void *base, int nxh, int n, int nfield, int ny, int KB, size_t es, CUtensorMap *m) {
  const EncodeTiledFn fn = encode_tiled();
  const int rows = tile_rows(n);
  if (!fn || 2 * KB > 256 || rows == 0 || (2 * KB * es) % 16 != 0 || (2 * (size_t)nxh * es) % 16 != 0 ||
      ((size_t)rows * KB * 2 * es) % 128 != 0 || (reinterpret_cast<uintptr_t>(base) & 15u) != 0)
    return false;
  const cuuint64_t dims[3] = {2ull * (cuuint64_t)nxh, (cuuint64_t)n, (cuuint64_t)nfield * (cuuint64_t)ny};
  const cuuint64_t strides[2] = {2ull * es * (cuuint64_t)nxh, 2ull * es * (cuuint64_t)nxh * (cuuint64_t)n};
  const cuuint32_t box[3] = {(cuuint32_t)(2 * KB), (cuuint32_t)rows, 1u}, ones[3] = {1u, 1u, 1u};
  return fn(m, es == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3,
            const_cast<void *>(base), dims, strides, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// y_to_x through TMA: only from the state S (the map covers its 3 + nsc fields)
template <typename R, int N1, int N2, int KB>
bool zinv_tma_map(const Handle &h, const double2 *src, int nfield, CUtensorMap *m) {
  return h.tune.ztma && src == h.S && nfield <= 3 + h.nsc &&
         z_smem_tma<R, N1, N2, KB, double2>(h.nz) <= (size_t)opt_in_smem() &&
         z_tile_map(h.S, h.nxh, h.nz, 3 + h.nsc, h.ny, KB, sizeof(double), m);
}

// x_to_y through TMA: only from the slab MID (the map covers its 5 + 3 nsc fields)
template <typename R, int N1, int N2, int KB>
bool zfwd_tma_map(const Handle &h, const void *mid, int nfield, CUtensorMap *m) {
  const int nprod = 5 + 3 * h.nsc;
  return h.tune.ztma && mid == h.MID && nfield <= nprod &&
         z_smem_tma<R, N1, N2, KB, typename Cpx<R>::T>(N1 * N2) <= (size_t)opt_in_smem() &&
         z_tile_map(h.MID, h.nxh, N1 * N2, nprod, h.ny, KB, sizeof(R), m);
}

// Returns cudaErrorNotSupported when the length has no four-step shape (caller falls back).
cudaError_t launch_zinv2(Handle &h, const double2 *src, void *mid, int nfield, cudaStream_t st, bool fp64) {
  cudaError_t err = cudaErrorNotSupported;
  auto go = [&]<typename R>() {
    with_shape(h.nz32, [&]<int N1, int N2>() {
      with_variant(h.tune.z, [&]<int V>() {
        using C = typename Cpx<R>::T;
        constexpr int KB = ZVar<R, tuned_variant<N1 * N2, V>()>::KB;
        dim3 grid((unsigned)((h.nxh + KB - 1) / KB), (unsigned)h.ny, (unsigned)nfield);
        CUtensorMap tmap{};
        if (zinv_tma_map<R, N1, N2, KB>(h, src, nfield, &tmap))
          k_zinv2<R, N1, N2, KB, true><<<grid, z_threads<N1, N2, KB>(), z_smem_tma<R, N1, N2, KB, double2>(h.nz),
                                         st>>>(src, reinterpret_cast<C *>(mid), h.pz, h.nz, h.nxh, h.ns, h.nm, tmap,
                                               h.ny, &h.dsc->err);
        else
          k_zinv2<R, N1, N2, KB, false><<<grid, z_threads<N1, N2, KB>(), z_smem<R, N1, N2, KB>(), st>>>(
              src, reinterpret_cast<C *>(mid), h.pz, h.nz, h.nxh, h.ns, h.nm, tmap, h.ny, &h.dsc->err);
        err = cudaGetLastError();
      });
    });
  };
  if (h.mixed && !fp64) go.template operator()<float>();
  else go.template operator()<double>();
  return err;
}

cudaError_t launch_zfwd2(Handle &h, const void *mid, void *dst, int nfield, double scale, bool dst_fp64,
                         cudaStream_t st, bool fp64) {
  cudaError_t err = cudaErrorNotSupported;
  auto go = [&]<typename R, typename D>() {
    with_shape(h.nz32, [&]<int N1, int N2>() {
      with_variant(h.tune.z, [&]<int V>() {
        using C = typename Cpx<R>::T;
        constexpr int KB = ZVar<R, tuned_variant<N1 * N2, V>()>::KB;
        dim3 grid((unsigned)((h.nxh + KB - 1) / KB), (unsigned)h.ny, (unsigned)nfield);
        CUtensorMap tmap{};
        if (zfwd_tma_map<R, N1, N2, KB>(h, mid, nfield, &tmap))
          k_zfwd2<R, N1, N2, KB, D, true><<<grid, z_threads<N1, N2, KB>(), z_smem_tma<R, N1, N2, KB, C>(N1 * N2),
                                            st>>>(reinterpret_cast<const C *>(mid), reinterpret_cast<D *>(dst), h.pz,
                                                  h.nz, h.nxh, h.ns, h.nm, scale, tmap, h.ny, &h.dsc->err);
        else
          k_zfwd2<R, N1, N2, KB, D, false><<<grid, z_threads<N1, N2, KB>(), z_smem<R, N1, N2, KB>(), st>>>(
              reinterpret_cast<const C *>(mid), reinterpret_cast<D *>(dst), h.pz, h.nz, h.nxh, h.ns, h.nm, scale,
              tmap, h.ny, &h.dsc->err);
        err = cudaGetLastError();
      });
    });
  };
  if (h.mixed && !fp64) {
    if (dst_fp64) go.template operator()<float, double2>();
    else go.template operator()<float, float2>();
  } else {
    go.template operator()<double, double2>();
  }
  return err;
}

bool z_tma_possible(const Handle &h, int zvar) {
  bool ok = false;
  auto go = [&]<typename R>() {
    with_shape(h.nz32, [&]<int N1, int N2>() {
      with_variant(zvar, [&]<int V>() {
        constexpr int KB = ZVar<R, tuned_variant<N1 * N2, V>()>::KB;
        CUtensorMap m{};
        ok = z_smem_tma<R, N1, N2, KB, double2>(h.nz) <= (size_t)opt_in_smem() &&
             z_tile_map(h.S, h.nxh, h.nz, 3 + h.nsc, h.ny, KB, sizeof(double), &m);
      });
    });
  };
  if (h.mixed) go.template operator()<float>();
  else go.template operator()<double>();
  return ok;
}

cudaError_t launch_xadj2(Handle &h, const double2 *base_mid, double2 *lmid, double scale, cudaStream_t st) {
  cudaError_t err = cudaErrorNotSupported;
  if (h.mixed) return err;
  with_shape(h.nx32, [&]<int N1, int N2>() {
    const dim3 grid((unsigned)h.nz32, (unsigned)h.ny);
    const size_t smem = sizeof(double2) * 6 * (size_t)ip_lda<N1, N2>();
    k_xadj2<N1, N2><<<grid, 128, smem, st>>>(base_mid, lmid, h.px, h.nz32, h.nxh, 1.0f / (float)h.nxh, h.nm, scale);
    err = cudaGetLastError();
  });
  return err;
}

void tile_shapes(const Handle &h, int zvar, int xvar, int *z_lines, int *x_rows, int *x_threads) {
  *z_lines = *x_rows = *x_threads = 0;
  auto zf = [&]<typename R>() {
    with_shape(h.nz32, [&]<int N1, int N2>() {
      with_variant(zvar, [&]<int V>() { *z_lines = ZVar<R, tuned_variant<N1 * N2, V>()>::KB; });
    });
    with_shape(h.nx32, [&]<int N1, int N2>() {
      with_variant(xvar, [&]<int V>() {
        using T = XVar<R, tuned_variant<N1 * N2, V>()>;
        *x_rows = T::ZB;
        *x_threads = T::ZT;
      });
    });
  };
  if (h.mixed) zf.template operator()<float>();
  else zf.template operator()<double>();
}

int xphys2_row_blocks(const Handle &h) {
  constexpr int zb = TCfg<double>::ZB;  // the statistics x pass computes in FP64 on every handle
  return (h.nz32 + zb - 1) / zb;
}

cudaError_t launch_xphys2(Handle &h, void *mid, int substep, cudaStream_t st, bool stat, double *mom) {
  cudaError_t err = cudaErrorNotSupported;
  X2Args a = x2_args(h, substep);
  a.mom = stat ? mom : nullptr;
  auto go = [&]<typename R>() {
    with_shape(h.nx32, [&]<int N1, int N2>() {
      using C = typename Cpx<R>::T;
      if constexpr (sizeof(R) == 8) {
        if (stat) {
          // the statistics variant keeps the default shape: its moment sums are laid out per row block
          using T = TCfg<R>;
          dim3 grid((unsigned)((h.nz32 + T::ZB - 1) / T::ZB), (unsigned)h.ny);
          k_xphys2<R, N1, N2, T::ZB, T::ZT, true><<<grid, T::ZT, x_smem<R, N1, N2>(), st>>>(reinterpret_cast<C *>(mid), h.px, a);
          err = cudaGetLastError();
          return;
        }
      }
      with_variant(h.tune.x, [&]<int V>() {
        constexpr int VV = tuned_variant<N1 * N2, V>();
        using T = XVar<R, VV>;
        dim3 grid((unsigned)((h.nz32 + T::ZB - 1) / T::ZB), (unsigned)h.ny);
        if (h.nsc == 2)
          k_xphys2<R, N1, N2, T::ZB, T::ZT, false, 2, VV><<<grid, T::ZT, x_smem<R, N1, N2, 2, T::ZB>(), st>>>(
              reinterpret_cast<C *>(mid), h.px, a);
        else
          k_xphys2<R, N1, N2, T::ZB, T::ZT, false, 1, VV><<<grid, T::ZT, x_smem<R, N1, N2, 1, T::ZB>(), st>>>(
              reinterpret_cast<C *>(mid), h.px, a);
        err = cudaGetLastError();
      });
    });
  };
  // the statistics products run in FP64 on every handle: a diagnostic off the step's path, whose
  // y derivatives of third moments and pressure covariances would carry FP32 rounding of the
  // physical velocities past 1e-5 of the line
  if (h.mixed && !stat) go.template operator()<float>();
  else go.template operator()<double>();
  return err;
}

}  // namespace kmm
