// transforms3.cu - the four-step transforms (transforms2.cuh) for the other common 3/2-padded lengths,
// those with a factor 5 or an uneven split, with one scalar.
//
// The generic mixed-radix kernels of transforms.cu pass a line through shared memory once a radix, with
// run-time radices and digit reversal: on 100x82x90 (lengths 150 and 135) FP64 they took 90 us (z inverse),
// 418 us (x pass) and 178 us (z forward) a substep.  Step only: the statistics, the pressure and the
// adjoint keep to transforms2.cu's lengths.
#include <cuda_runtime.h>

#include "transforms2.cuh"

namespace kmm {

namespace {

template <typename F> bool with_other_shape(int N, F &&f) {
  switch (N) {
    case 27: f.template operator()<3, 9>(); return true;
    case 30: f.template operator()<5, 6>(); return true;
    case 45: f.template operator()<5, 9>(); return true;
    case 54: f.template operator()<6, 9>(); return true;
    case 60: f.template operator()<6, 10>(); return true;
    case 75: f.template operator()<5, 15>(); return true;
    case 81: f.template operator()<9, 9>(); return true;
    case 90: f.template operator()<9, 10>(); return true;
    case 108: f.template operator()<9, 12>(); return true;
    case 120: f.template operator()<10, 12>(); return true;
    case 135: f.template operator()<9, 15>(); return true;
    case 150: f.template operator()<10, 15>(); return true;
    case 162: f.template operator()<9, 18>(); return true;
    case 180: f.template operator()<12, 15>(); return true;
    case 216: f.template operator()<12, 18>(); return true;
    case 225: f.template operator()<15, 15>(); return true;
    case 240: f.template operator()<15, 16>(); return true;
    case 243: f.template operator()<9, 27>(); return true;
    case 270: f.template operator()<15, 18>(); return true;
    case 300: f.template operator()<15, 20>(); return true;
    case 324: f.template operator()<18, 18>(); return true;
    case 360: f.template operator()<18, 20>(); return true;
    case 375: f.template operator()<15, 25>(); return true;
    case 432: f.template operator()<18, 24>(); return true;
    case 480: f.template operator()<20, 24>(); return true;
    default: return false;
  }
}

}  // namespace

// Shared-memory limits of the kernels h's lengths use (setting all 25 lengths' took 1 ms of kmm_create).
cudaError_t prepare_transforms3(const Handle &h) {
  cudaError_t e = cudaSuccess;
  using D = TCfg<double>;
  using F = TCfg<float>;
  bool used = with_other_shape(h.nz32, [&]<int N1, int N2>() {
    set_smem(k_zinv2<double, N1, N2, D::KB>, h.smem_optin);
    set_smem(k_zinv2<float, N1, N2, F::KB>, h.smem_optin);
    set_smem(k_zfwd2<double, N1, N2, D::KB, double2>, h.smem_optin);
    set_smem(k_zfwd2<float, N1, N2, F::KB, float2>, h.smem_optin);
    set_smem(k_zfwd2<float, N1, N2, F::KB, double2>, h.smem_optin);
  });
  used |= with_other_shape(h.nx32, [&]<int N1, int N2>() {
    set_smem(k_xphys2<double, N1, N2, D::ZB, D::ZT>, h.smem_optin);
    set_smem(k_xphys2<float, N1, N2, F::ZB, F::ZT>, h.smem_optin);
  });
  if (used) e = fill_regtw();
  return e;
}

// Each returns cudaErrorNotSupported for other lengths (the caller falls back).
cudaError_t launch_zinv3(Handle &h, const double2 *src, void *mid, int nfield, cudaStream_t st, bool fp64) {
  cudaError_t err = cudaErrorNotSupported;
  auto go = [&]<typename R>() {
    with_other_shape(h.nz32, [&]<int N1, int N2>() {
      constexpr int KB = TCfg<R>::KB;
      const dim3 grid((unsigned)((h.nxh + KB - 1) / KB), (unsigned)h.ny, (unsigned)nfield);
      k_zinv2<R, N1, N2, KB><<<grid, z_threads<N1, N2, KB>(), z_smem<R, N1, N2, KB>(), st>>>(
          src, reinterpret_cast<typename Cpx<R>::T *>(mid), h.pz, h.nz, h.nxh, h.ns, h.nm, CUtensorMap{}, h.ny,
          &h.dsc->err);
      err = cudaGetLastError();
    });
  };
  if (h.mixed && !fp64) go.template operator()<float>();
  else go.template operator()<double>();
  return err;
}

cudaError_t launch_zfwd3(Handle &h, const void *mid, void *dst, int nfield, double scale, bool dst_fp64,
                         cudaStream_t st, bool fp64) {
  cudaError_t err = cudaErrorNotSupported;
  auto go = [&]<typename R, typename D>() {
    with_other_shape(h.nz32, [&]<int N1, int N2>() {
      constexpr int KB = TCfg<R>::KB;
      const dim3 grid((unsigned)((h.nxh + KB - 1) / KB), (unsigned)h.ny, (unsigned)nfield);
      k_zfwd2<R, N1, N2, KB, D><<<grid, z_threads<N1, N2, KB>(), z_smem<R, N1, N2, KB>(), st>>>(
          reinterpret_cast<const typename Cpx<R>::T *>(mid), reinterpret_cast<D *>(dst), h.pz, h.nz, h.nxh, h.ns, h.nm,
          scale, CUtensorMap{}, h.ny, &h.dsc->err);
      err = cudaGetLastError();
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

cudaError_t launch_xphys3(Handle &h, void *mid, int substep, cudaStream_t st) {
  cudaError_t err = cudaErrorNotSupported;
  if (h.nsc != 1) return err;
  const X2Args a = x2_args(h, substep);
  auto go = [&]<typename R>() {
    with_other_shape(h.nx32, [&]<int N1, int N2>() {
      using T = TCfg<R>;
      const dim3 grid((unsigned)((h.nz32 + T::ZB - 1) / T::ZB), (unsigned)h.ny);
      k_xphys2<R, N1, N2, T::ZB, T::ZT><<<grid, T::ZT, x_smem<R, N1, N2>(), st>>>(
          reinterpret_cast<typename Cpx<R>::T *>(mid), h.px, a);
      err = cudaGetLastError();
    });
  };
  if (h.mixed) go.template operator()<float>();
  else go.template operator()<double>();
  return err;
}

}  // namespace kmm
