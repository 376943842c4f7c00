// mean.cu - the mean lines of one substep (wave00.f90:41-714).
#include <cuda_runtime.h>

#include "kmm_internal.h"
#include "lines.cuh"

namespace kmm {

namespace {

// ------------------------------------------------------------------------------------------
// k_mean: wave00.f90 for the mean lines: U (line 0: forced, Galilean shift), W (line 1: phi = 0), Theta
// (line 2: nu/pr, forced to the bulk value), a second scalar (line 3).  One block; warp l holds line l
// in shared memory, its serial chains (real and imaginary parts, flux and store) a lane each and the
// rest over all lanes, while warp 4 + l factors the line's operator.  One thread a line, with its work
// lines in global memory, took 464 us at ny = 129, longer than the solver kernels beside it; this takes 134.
struct MeanArgs {
  int ny, substep, nsc;
  int64_t nmodes, ns;
  double2 *S, *RK;
  const void *P;
  bool mixed;    // P holds float2
  double *w00;   // the lines where shared memory cannot hold them
  const double *tabs, *tt, *integ;
  double nu, pr, bulk_u, bulk_w, bulk_t, u_gal;
  double pr2, bulk_t2;  // a second passive scalar (line 3)
  DevScalars *dsc;
  const double *dt_ptr;
};

// One line's LU, 0-based rows: l[r][BW+1] = 1 / L(r, r), L(r, r-d) / L(r, r); lx the same for d > BW of the
// last BW rows; u[r][BW] = U(r, r+e); ux for e > BW of the first BW rows.
template <int BW>
struct MeanLu {
  double *l, *lx, *u, *ux;
  // LuSweep's U store (1-based rows)
  __device__ __forceinline__ double get(int r, int e) const {
    if (e <= BW) return u[(r - 1) * BW + e - 1];
    return r <= BW ? ux[(r - 1) * BW + e - BW - 1] : 0.0;
  }
  __device__ __forceinline__ void set(int r, int e, double v) const {
    if (e <= BW) u[(r - 1) * BW + e - 1] = v;
    else if (r <= BW) ux[(r - 1) * BW + e - BW - 1] = v;
  }
};

// Doubles of a line: eight real planes, then its LU.
__host__ __device__ constexpr int64_t mean_line_doubles(int bw, int n) {
  return (int64_t)n * (8 + 2 * bw + 1) + 2 * bw * bw;
}

template <int BW, bool SM>
__global__ void __launch_bounds__(256) k_mean(MeanArgs a) {
  extern __shared__ double mean_smem[];
  if (block_failed(a.dsc)) return;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, line = warp % 4;
  const bool mine = line < 2 + a.nsc;
  const int n = a.ny, s = a.substep;
  const int64_t ns = a.ns;
  const double dt = *a.dt_ptr;
  // line 3: a second passive scalar, the theta block with its own Prandtl number and bulk value
  const double visc = (line == 2) ? a.nu / a.pr : (line == 3) ? a.nu / a.pr2 : a.nu;
  const double gal = (line == 0) ? a.u_gal : 0.0;
  double *base = (SM ? mean_smem : a.w00) + (int64_t)line * mean_line_doubles(BW, n);
  // planes: the flux product re, im; the store re, im; D1 D0^{-1} flux re, im; the solve's re, im
  double *F = base, *Z = F + 2 * n, *DF = Z + 2 * n, *R = DF + 2 * n;
  MeanLu<BW> lu;
  lu.l = R + 2 * n;
  lu.u = lu.l + n * (BW + 1);
  lu.lx = lu.u + n * BW;
  lu.ux = lu.lx + BW * BW;
  const Tabs<BW> tb = tabs_at<BW>(a.tabs, n);
  const DLine store{a.RK + line * ns, a.nmodes};
  auto dot = [&](int d, const double *x, int r) {  // row r of D_d times the coefficients x
    const double *t = row_entries<BW>(a.tt, r) + d;
    const double *y = x + first_col<BW>(r, n);
    double acc = 0.0;
#pragma unroll
    for (int j = 0; j <= 2 * BW; ++j) acc += t[3 * j] * y[j];
    return acc;
  };
  if (warp >= 4) {
    if (mine && lane == 0) {  // (D0 - beta D2), Dirichlet rows
      const double beta = dt * rkc(2, s) * visc;
      LuSweep<BW, 0, 0, true, MeanLu<BW>> sweep;
      sweep.init(n, lu);
      const double2 bc[1] = {z2(0.0, 0.0)};
      const double br[1] = {0.0};
      double2 zc[1];
      double zr[1];
      for (int r = 1; r <= n; ++r) {
        sweep.step(r, [&](int rr, double *row, bool c) { helm_row<BW>(tb, rr, n, 1.0, beta, row, c); }, bc, br, zc, zr);
        double *l = lu.l + (r - 1) * (BW + 1);
        l[0] = sweep.Lk[0];
#pragma unroll
        for (int d = 1; d <= BW; ++d) l[d] = sweep.Lk[d] * sweep.Lk[0];
        if (r > n - BW) {
#pragma unroll
          for (int d = BW + 1; d <= 2 * BW; ++d) lu.lx[(r - 1 - (n - BW)) * BW + d - BW - 1] = sweep.Lk[d] * sweep.Lk[0];
        }
      }
    }
  } else if (mine) {
    const int pslot = (line == 0) ? 1 : (line == 1) ? 3 : (line == 2) ? 6 : 9;  // uv, vw, v theta, v theta2
    auto prod = [&](int r) {
      const int64_t o = pslot * ns + (int64_t)r * a.nmodes;
      return a.mixed ? ldp<float2>(reinterpret_cast<const float2 *>(a.P) + o)
                     : ldp<double2>(reinterpret_cast<const double2 *>(a.P) + o);
    };
    for (int r = lane; r < n; r += 32) {
      const double2 f = prod(r), z = store.ld(r + 1);
      F[r] = f.x;
      F[n + r] = f.y;
      Z[r] = z.x;
      Z[n + r] = z.y;
    }
    __syncwarp();
    // D0 solves: the flux product (and the store at substep 1)
    if (lane < (s == 1 ? 4 : 2)) {
      double *x = F + lane * n;
      fixed_fwd<BW, 1>(x, n, [&](int r, int d) { return tb.l0[r * (2 * BW + 1) + d] * tb.l0[r * (2 * BW + 1)]; },
                   [&](int r) { return tb.l0[r * (2 * BW + 1)]; });
      fixed_bwd<BW, 1>(x, n, [&](int r, int e) { return tb.u0[r * 2 * BW + e - 1]; });
    }
    __syncwarp();
    const double gamma = dt * rkc(3, s), alpha = dt * rkc(1, s) * visc;
    for (int r = lane; r < n; r += 32) {
      const double dx = dot(1, F, r), dy = dot(1, F + n, r);  // d/dy of the flux
      DF[r] = dx;
      DF[n + r] = dy;
      double b = store.ld(r + 1).x;
      if (s == 1) b += alpha * dot(2, Z, r);
      b -= gamma * dx;
      // wave00.f90:169-173: zero wall rows, interior real part + u_gal, imaginary part 1
      const bool wall = r == 0 || r == n - 1;
      R[r] = wall ? 0.0 : b + gal;
      R[n + r] = wall ? 0.0 : 1.0;
    }
  }
  __syncthreads();
  if (warp >= 4 || !mine) return;
  if (lane < 2) {
    double *x = R + lane * n;
    fixed_fwd<BW, 1>(x, n,
                 [&](int r, int d) {
                   return d <= BW ? lu.l[r * (BW + 1) + d] : lu.lx[(r - (n - BW)) * BW + d - BW - 1];
                 },
                 [&](int r) { return lu.l[r * (BW + 1)]; });
    fixed_bwd<BW, 1>(x, n, [&](int r, int e) { return e <= BW ? lu.u[r * BW + e - 1] : lu.ux[r * BW + e - BW - 1]; });
  }
  __syncwarp();
  // LABS_integration of the coefficients, real and imaginary part
  double ix = 0.0, iy = 0.0;
  for (int r = lane; r < n; r += 32) {
    ix += __ldg(a.integ + r) * R[r];
    iy += __ldg(a.integ + r) * R[n + r];
  }
  for (int o = 16; o > 0; o >>= 1) {
    ix += __shfl_xor_sync(0xffffffffu, ix, o);
    iy += __shfl_xor_sync(0xffffffffu, iy, o);
  }
  const double bulk = (line == 0) ? a.bulk_u : (line == 1) ? a.bulk_w : (line == 2) ? a.bulk_t : a.bulk_t2;
  double phi = (bulk - 0.5 * ix) / (0.5 * iy);  // calculate_phi
  if (line == 1) phi = 0.0;                     // wave00.f90:396
  // c = Re c + phi Im c (real)
  for (int r = lane; r < n; r += 32) R[r] += phi * R[n + r];
  __syncwarp();
  if (lane == 0) {
    if (s == 3) {
      const double *r1 = trow<BW>(tb.t1, 1), *rn = trow<BW>(tb.t1, n);
      const double wall = r1[0] * R[0] + r1[1] * R[1] - rn[-1] * R[n - 2] - rn[0] * R[n - 1];
      if (line == 0) a.dsc->wall_shear_stress = 0.5 * a.nu * wall;
      if (line == 2) a.dsc->wall_theta_stress = 0.5 * a.nu / a.pr * wall;
      if (line == 3) a.dsc->wall_theta_stress2 = 0.5 * a.nu / a.pr2 * wall;
    }
    if (line == 0) a.dsc->phi_dpdx[s - 1] = phi;
    if (line == 2) a.dsc->phi_dtdx[s - 1] = phi;
    if (line == 3) a.dsc->phi_dtdx2[s - 1] = phi;
  }
  const DLine out{a.S + (line == 0 ? 0 : line == 1 ? 2 : line == 2 ? 3 : 4) * ns, a.nmodes};
  const DLine Sv{a.S + ns, a.nmodes};
  for (int r = lane; r < n; r += 32) {
    const double prof = dot(0, R, r) - gal;
    out.st(r + 1, z2(prof, 0.0));
    double2 st = z2(prof, 0.0);
    if (s != 3) {
      const double alpha = dt * rkc(1, s + 1) * visc, zeta = dt * rkc(4, s + 1);
      st = z2(alpha * dot(2, R, r) + prof - zeta * DF[r], -zeta * DF[n + r]);
    }
    store.st(r + 1, st);
    if (line == 1) Sv.st(r + 1, z2(0.0, 0.0));  // v mean = 0 (wave00.f90:462)
  }
}

template <int BW>
cudaError_t mean_bw(Handle &h, int substep, const double *dt_ptr, cudaStream_t st) {
  const OpsOffsets off = ops_offsets(h.bw, h.ny);
  MeanArgs ma;
  ma.ny = h.ny;
  ma.substep = substep;
  ma.nsc = h.nsc;
  ma.pr2 = h.cfg.pr2;
  ma.bulk_t2 = h.cfg.bulk_t2;
  ma.nmodes = h.nmodes;
  ma.ns = h.ns;
  ma.S = h.S;
  ma.RK = h.RK;
  ma.P = h.P;
  ma.w00 = h.w00;
  ma.tabs = h.dops + off.t0;
  ma.tt = h.dops + off.tt;
  ma.integ = h.dops + off.integ;
  ma.nu = h.cfg.nu;
  ma.pr = h.cfg.pr;
  ma.bulk_u = h.cfg.bulk_vel_u;
  ma.bulk_w = h.cfg.bulk_vel_w;
  ma.bulk_t = h.cfg.bulk_t;
  ma.u_gal = h.cfg.u_gal;
  ma.dsc = h.dsc;
  ma.dt_ptr = dt_ptr;
  ma.mixed = h.mixed;
  const size_t bytes = sizeof(double) * (size_t)mean_doubles(h);
  if (bytes <= (size_t)h.smem_optin) k_mean<BW, true><<<1, 256, bytes, st>>>(ma);
  else k_mean<BW, false><<<1, 256, 0, st>>>(ma);  // ny above about 400
  return cudaGetLastError();
}

template <int BW>
cudaError_t limit_bw(int bytes) {
  return cudaFuncSetAttribute(k_mean<BW, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

}  // namespace

int64_t mean_doubles(const Handle &h) { return (2 + h.nsc) * mean_line_doubles(h.bw, h.ny); }

cudaError_t prepare_mean(Handle &h) {
  switch (h.bw) {
    case 2: return limit_bw<2>(h.smem_optin);
    case 3: return limit_bw<3>(h.smem_optin);
    case 4: return limit_bw<4>(h.smem_optin);
    case 5: return limit_bw<5>(h.smem_optin);
    case 6: return limit_bw<6>(h.smem_optin);
    case 7: return limit_bw<7>(h.smem_optin);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_mean(Handle &h, int substep, const double *dt_ptr, cudaStream_t st) {
  switch (h.bw) {
    case 2: return mean_bw<2>(h, substep, dt_ptr, st);
    case 3: return mean_bw<3>(h, substep, dt_ptr, st);
    case 4: return mean_bw<4>(h, substep, dt_ptr, st);
    case 5: return mean_bw<5>(h, substep, dt_ptr, st);
    case 6: return mean_bw<6>(h, substep, dt_ptr, st);
    case 7: return mean_bw<7>(h, substep, dt_ptr, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace kmm
