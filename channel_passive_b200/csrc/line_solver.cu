// line_solver.cu - the Helmholtz solves of one substep (solve_t.f90:28-201, solve_g.f90:28-201,
// solve_v_f.f90:38-375) and the velocities they give (solve_u_w.f90:18-42), one block per tile of modes.
//
//   k_line_factor     the operators' LU per mode, in TileFac layout: theta's (alpha D0 - beta_t D2), the one
//                g and phi share, a second scalar's, and once per handle v's (D2 - k^2 D0).
//   k_lines  right-hand sides into shared memory; the chains theta, g, phi_p (re, im) and phi_h
//                through their factors; theta and phi formed; v_p and v_h through v's factors; then
//                C1, C2 (solve_v_f.f90:293-298), v, dv/dy, the stores, u and w.
#include <cuda_runtime.h>

#include "kmm_internal.h"
#include "lines.cuh"

namespace kmm {

namespace {

struct HelmArgs {
  int n, nxh, nz, substep;
  int64_t nmodes, ns;
  // lines of the state and the stores, and k_hvhg's (HLine; H_HV0..H_V3 and H_HT2 at the products'
  // type): one pointer each, because the addresses then come from constant operands and take no registers
  double2 *S[5], *RK[4];
  const void *hl[H_COUNT];
  const double *tabs;       // T0, T1, T2 [n][4BW+1]
  const double *tt;         // their rows as the mat-vecs read them (row_entries)
  const double2 *vwall;     // [2][nm] control probes v(y_d), v(-y_d) of each mode
  const float *gains;       // control gain per mode
  double control_amp;
  double nu, pr, pr2, lmfxr, lmfzr;
  DevScalars *dsc;
  const double *dt_ptr;
  double *fac[3];           // TileFac sets of theta, of g and phi, and of a second scalar
  double *vf;               // of v
  double *fcdt;             // the dt the sets fac hold (a fixed time step), or null
  unsigned *fcount;         // blocks of k_line_factor done with them
  bool cached;              // the sets may be kept while they hold this dt (Tuning::fcache)
  int stages;               // ring slots
};

// ------------------------------------------------------------------------------------------
// k_line_factor: one thread per mode and operator; op = blockIdx.y (0 theta, 1 g and phi, 2 theta2), or
// v's operator with a.fac[0] null.  LuSweep's profile Crout LU, stored by tile.  A no-op while the
// sets hold this dt (a fixed time step: 3 us against 117 us on 128x97x128 once a substep and run).
// The sets and the dt they hold are written here together, by the last block to finish: it runs beside the
// transforms, and whatever becomes of the substep after it, the mark is that of the sets.  (For the same
// reason it does not look at the error flag: some blocks would leave and others not.)
template <int BW>
__global__ void __launch_bounds__(32) k_line_factor(HelmArgs a) {
  const bool vop = a.fac[0] == nullptr;
  if (!vop && a.cached && *a.fcdt == *a.dt_ptr) return;
  const int64_t m = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= a.nmodes) return;
  const int n = a.n, op = blockIdx.y;
  const Tabs<BW> tb = tabs_at<BW>(a.tabs, n);
  const double k2 = mode_k((int)m, a.nxh, a.nz, a.lmfxr, a.lmfzr).k2;
  double *f = (vop ? a.vf : a.fac[op]) + (m / kTile) * TileFac<BW>::size(n);
  const int km = (int)(m % kTile);
  double ca = 0.0, cb = 0.0;
  if (!vop) {
    cb = *a.dt_ptr * rkc(2, a.substep) * (op == 0 ? a.nu / a.pr : op == 1 ? a.nu : a.nu / a.pr2);
    ca = 1.0 + cb * k2;
  }
  LuSweep<BW, 0, 0, true, TileU<BW>> lu;
  lu.init(n, TileU<BW>{f + TileFac<BW>::bwd(n), f + TileFac<BW>::bx(n) + km, n, km});
  const double2 bc[1] = {z2(0.0, 0.0)};
  const double br[1] = {0.0};
  double2 zc[1];
  double zr[1];
  for (int r = 1; r <= n; ++r) {
    lu.step(r, [&](int rr, double *row, bool c) {
      if (vop) vrow<BW>(tb, rr, n, k2, row, c);
      else helm_row<BW>(tb, rr, n, ca, cb, row, c);
    }, bc, br, zc, zr);
    const int q = r - 1;  // 0-based
    auto entry = [&](int row, int k) -> double & { return f[(int64_t)row * (BW + 1) * kTile + entry_at(BW + 1, k, km)]; };
    if (q >= BW) entry(q - BW, 0) = lu.Lk[0];
    else f[TileFac<BW>::fx(n) + (BW * BW + q) * kTile + km] = lu.Lk[0];
#pragma unroll
    for (int d = 1; d <= BW; ++d)
      if (q >= d) entry(q - d, d) = lu.Lk[d] * lu.Lk[0];
    if (q >= n - BW) {
      double *x = f + TileFac<BW>::fx(n) + (q - (n - BW)) * BW * kTile + km;
#pragma unroll
      for (int d = BW + 1; d <= 2 * BW; ++d) x[(d - BW - 1) * kTile] = lu.Lk[d] * lu.Lk[0];
    }
  }
  // thread 0 of every block has a mode; every block has read the old mark by the time it counts
  if (!vop && a.fcdt && threadIdx.x == 0 && atomicAdd(a.fcount, 1u) + 1 == gridDim.x * gridDim.y) {
    *a.fcount = 0;
    *a.fcdt = *a.dt_ptr;
  }
}

// ------------------------------------------------------------------------------------------
// Planes of a block (real, [row][mode]): theta re, im; g re, im; phi re, im; phi_h; v_h; with a
// second scalar theta2 re, im.  v_p takes theta's two once theta is done.
enum Plane { P_T = 0, P_G = 2, P_PHI = 4, P_PHIH = 6, P_VH = 7, P_T2 = 8 };
constexpr int helm_planes(int nsc) { return 8 + 2 * (nsc - 1); }
// The chain threads, in whole warps: 7 chains of kTile modes, 9 with a second scalar.
constexpr int helm_chain_threads(int nsc) { return ((5 + 2 * nsc) * kTile + 31) / 32 * 32; }
// Two blocks of eight warps an SM (128 registers a thread), 16 modes in flight.  Tiles of 4 modes in 3 or 4
// blocks an SM were slower (64x65x64: 57 against 41 us, its 512 tiles take two waves), and so were shapes that
// spilled more than these registers do (128 to 208 bytes at BW = 4): local memory finds no L1 beside the lines.
// Above ny = 139 at BW = 4 (79 with two scalars) one block is resident.  64x65x64 FP64: 38 us with k_line_factor's
// no-op, against 147 + 12 with k_helmholtz and k_assemble; 128x97x128 162 against 238 + 29.
constexpr int kHelmThreads = 256;
constexpr int kHelmBlocks = 2;  // resident blocks asked for

template <int BW, int NS>
struct HelmSmem {
  static constexpr int NOP = 1 + NS;
  static constexpr int slot = NOP * slot_rows<BW>() * (BW + 1) * kTile;  // doubles of a ring slot
  static constexpr int ext = TileFac<BW>::ext;                  // doubles of one fx or bx block
  static __host__ __device__ constexpr int plane(int n) { return (n | 1) * kTile; }
  static constexpr size_t bytes(int n, int stages) {
    return sizeof(double) * (size_t)(stages * slot + (NOP + 1) * 2 * ext + 4 * kTile + 2 * kMaxStages + 2 +
                                     helm_planes(NS) * plane(n));
  }
};

// PT the products' type of k_hvhg's lines, NS scalars.
template <int BW, typename PT, int NS>
__global__ void __launch_bounds__(kHelmThreads, kHelmBlocks) k_lines(HelmArgs a) {
  using L = HelmSmem<BW, NS>;
  constexpr int NOP = L::NOP, NP = helm_planes(NS), CT = helm_chain_threads(NS);
  extern __shared__ __align__(128) double helm_smem[];
  if (block_failed(a.dsc)) return;
  const int n = a.n, s = a.substep, tid = threadIdx.x;
  const int nm = (int)a.nmodes, ps = L::plane(n);  // (a line has fewer than 2^31 elements)
  // outside the chains a thread works on one mode, in rows RT apart
  constexpr int RT = kHelmThreads / kTile;
  const int m = blockIdx.x * kTile + tid % kTile;
  const bool live = m > 0 && m < nm;  // (mode 0 is k_mean's, beside this kernel)
  const int k = tid % kTile, rt = tid / kTile;
  const ModeK kk = mode_k(live ? (int)m : 0, a.nxh, a.nz, a.lmfxr, a.lmfzr);
  const double k2 = kk.k2;
  double *pl = helm_smem, *ring = pl + NP * ps;
  const int S = a.stages;
  double *ext = ring + S * L::slot;        // [op: theta, g, (theta2,) v][fx, bx]
  double *cc = ext + (NOP + 1) * 2 * L::ext;     // C1, C2 per mode
  uint64_t *bar = reinterpret_cast<uint64_t *>(cc + 4 * kTile);
  const double dt = *a.dt_ptr, nu = a.nu;
  const int C = sweep_chunks<BW>(n);             // chunks of a sweep

  // ---- the staged factor chunks, in the order the chains read them: ops 0..NOP-1 forward (C
  // chunks), backward (C, descending), then v forward and backward
  auto op_set = [&](int op) {
    const double *base = op == NOP ? a.vf : a.fac[op];
    return base + blockIdx.x * TileFac<BW>::size(n);
  };
  // Producer lane o copies operator o's chunks (in v's sweeps lane 0 alone); a slot is filled again
  // once every chain warp has arrived on its empty barrier.  Lanes of one warp, because a copy takes a
  // few hundred cycles to issue: in a chain's own warp it was a third of the sweep.
  uint64_t *full = bar, *empty = bar + kMaxStages, *extb = bar + 2 * kMaxStages, *rowb = extb + 1;
  auto issue = [&](int g, int slot, int lane) {
    const bool v = g >= 2 * C;
    const int q = v ? g - 2 * C : g, W = q < C ? BW + 1 : BW, c = q < C ? q : 2 * C - 1 - q;
    const unsigned bytes = (unsigned)(chunk_rows(c, C, n) * W * kTile * sizeof(double));
    const int on = v ? 1 : NOP;
    if (lane == 0) mbar_expect_tx(full + slot, on * bytes);
    __syncwarp();
    if (lane < on)
      bulk_load(ring + slot * L::slot + lane * slot_rows<BW>() * W * kTile,
                op_set(v ? NOP : lane) + (q < C ? 0 : TileFac<BW>::bwd(n)) + (int64_t)c * kChunk * W * kTile, bytes,
                full + slot);
  };
  if (tid == 0) {
    for (int i = 0; i < S; ++i) {
      mbar_init(full + i, 1);
      mbar_init(empty + i, CT / 32);
    }
    mbar_init(extb, 1);
    mbar_init(rowb, 1);
    mbar_expect_tx(extb, (unsigned)((NOP + 1) * 2 * L::ext * sizeof(double)));
  }
  __syncthreads();
  const bool producer = tid >= kHelmThreads - 32;
  if (producer) {
    const int lane = tid % 32;
    if (lane < 2 * (NOP + 1))
      bulk_load(ext + lane * L::ext, op_set(lane / 2) + (lane % 2 == 0 ? TileFac<BW>::fx(n) : TileFac<BW>::bx(n)),
                L::ext * sizeof(double), extb);
    for (int g = 0; g < S && g < 4 * C; ++g) issue(g, g, lane);
  }

  // ---- right-hand sides (solve_g.f90:84-123); rows 0 and n-1 are the Dirichlet rows (zero)
  auto hp = [&](int i) { return reinterpret_cast<const PT *>(a.hl[i]); };
  auto h_of = [&](int i, int o) { const PT v = ld_stream(hp(i) + o); return z2((double)v.x, (double)v.y); };
  const double visc_t = nu / a.pr, visc_t2 = NS == 2 ? nu / a.pr2 : 0.0;
  const double a1 = dt * rkc(1, s), gamma = dt * rkc(3, s);
  const double p0 = (1.0 + dt * rkc(2, s) * nu * k2) * a.tt[0] - dt * rkc(2, s) * nu * a.tt[2];  // A_g(1,1)
  const int ml = live ? m : 0;  // (a lane without a mode loads mode 0 and keeps nothing)
  constexpr int NST = 2 + NS;
  constexpr int store_of[4] = {2, 0, 1, 3}, d2_of[4] = {H_DT, H_DG, H_DP, H_DT2};  // theta, g, phi, theta2
  constexpr int LR = 2;  // rows whose loads a thread has in flight together
  for (int rb = rt; rb < n; rb += LR * RT) {
    double2 st[LR][NST], d2[LR][NST];
    PT hh[LR][4];
#pragma unroll
    for (int q = 0; q < LR; ++q) {
      const int o = min(rb + q * RT, n - 1) * nm + ml;
#pragma unroll
      for (int i = 0; i < NST; ++i) {
        st[q][i] = ld_stream(a.RK[store_of[i]] + o);
        if (s == 1) d2[q][i] = ld_stream(reinterpret_cast<const double2 *>(a.hl[d2_of[i]]) + o);
      }
      hh[q][0] = ld_stream(hp(H_HT) + o);
      hh[q][1] = ld_stream(hp(H_G2) + o);
      hh[q][2] = ld_stream(hp(H_HV0) + o);
      if constexpr (NS == 2) hh[q][3] = ld_stream(hp(H_HT2) + o);
    }
#pragma unroll
    for (int q = 0; q < LR; ++q) {
      const int r = rb + q * RT;
      if (r >= n) break;
      const bool in = live && r > 0 && r < n - 1;
      auto wide = [&](int i) { return z2((double)hh[q][i].x, (double)hh[q][i].y); };
      const double2 h[4] = {wide(0), wide(1), wide(2), NS == 2 ? wide(3) : z2(0.0, 0.0)};
      double *x = pl + r * kTile + k;
#pragma unroll
      for (int i = 0; i < NST; ++i) {
        double2 v = zscale(gamma, h[i]);
        if (s == 1) {
          const double alpha = a1 * (i == 0 ? visc_t : i == 3 ? visc_t2 : nu);
          v = zadd(zadd(zscale(1.0 - alpha * k2, st[q][i]), v), zscale(alpha, d2[q][i]));
        } else {
          v = zadd(st[q][i], v);
        }
        if (!in) v = z2(0.0, 0.0);
        const int plane = i == 0 ? P_T : i == 1 ? P_G : i == 2 ? P_PHI : P_T2;
        x[plane * ps] = v.x;
        x[(plane + 1) * ps] = v.y;
      }
      x[P_PHIH * ps] = r == 0 ? p0 : 0.0;  // the unit-wall right-hand side A_g(1,1) e_1 (solve_v_f.f90:140-153)
    }
  }
  __syncthreads();

  // ---- the chains: thread (chain, mode) of the first CT threads
  bool ok = true;
  int slot = 0;        // the ring slot and phase of this thread's next chunk (chains and producer alike)
  unsigned phase = 0;
  auto advance = [&]() {
    if (++slot == S) {
      slot = 0;
      phase ^= 1;
    }
  };
  const int chain = tid / kTile, cm = tid % kTile;
  auto sweeps = [&](int plane, int op, int ring_op, bool active) {
    const unsigned x = smem_u32(pl + plane * ps + cm);
    const unsigned fx = smem_u32(ext + 2 * op * L::ext + cm), bx = fx + 8u * L::ext;
    double acc[BW];
#pragma unroll
    for (int i = 0; i < BW; ++i) acc[i] = 0.0;
    for (int q = 0; q < 2 * C; ++q) {
      if (ok) ok = mbar_wait_bounded(full + slot, phase);
      if (active) {
        const unsigned co =
            smem_u32(ring + slot * L::slot + ring_op * slot_rows<BW>() * (q < C ? BW + 1 : BW) * kTile);
        if (q < C) fwd_chunk<BW>(x, co, fx, cm, q, C, n, acc);
        else bwd_chunk<BW>(x, co, bx, cm, 2 * C - 1 - q, C, n, acc);
      }
      __syncwarp();  // the warp's chains are done with the slot
      if (tid % 32 == 0) mbar_arrive(empty + slot);
      advance();
    }
  };
  // the producer's part of the two sweeps from chunk `first` on
  auto feed = [&](int first) {
    for (int g = first; g < first + 2 * C && g + S < 4 * C; ++g) {
      if (ok) ok = mbar_wait_bounded(empty + slot, phase);
      if (!__all_sync(0xffffffffu, ok)) {
        ok = false;
        break;
      }
      issue(g + S, slot, tid % 32);
      advance();
    }
  };
  // leaves after a wait that gave up: the copies still in flight get one more bounded wait each
  auto leave = [&]() {
    if (tid == 0) {
      atomicCAS(&a.dsc->err, 0, KMM_ERR_TIMEOUT);
      for (int i = 0; i < S; ++i) {
        mbar_wait_bounded(full + i, 0);
        mbar_wait_bounded(full + i, 1);
      }
      mbar_wait_bounded(extb, 0);
      mbar_wait_bounded(rowb, 0);
      mbar_wait_bounded(rowb, 1);
    }
    __syncthreads();
  };
  if (tid < CT) {
    ok = mbar_wait_bounded(extb, 0);
    const bool active = chain < 7 + 2 * (NS - 1);
    const int plane = chain < 7 ? chain : P_T2 + chain - 7, op = chain < 2 ? 0 : chain < 7 ? 1 : 2;
    sweeps(active ? plane : 0, active ? op : 0, active ? op : 0, active);
  } else if (producer) {
    feed(0);
  }
  if (__syncthreads_or(!ok)) {
    leave();
    return;
  }

  // new store (solve_g.f90:138-185): zeta' h + (1 - alpha' k2) f + alpha' D2 f, or f at s = 3
  const double a1n = s == 3 ? 0.0 : dt * rkc(1, s + 1), zeta = s == 3 ? 0.0 : dt * rkc(4, s + 1);
  auto store_new = [&](double2 h, double2 f, double2 d2f, double visc) {
    if (s == 3) return f;
    const double alpha = a1n * visc;
    return zadd(zadd(zscale(zeta, h), zscale(1.0 - alpha * k2, f)), zscale(alpha, d2f));
  };

  // ---- the scalars from their coefficients
  if (live)
    for (int r = rt; r < n; r += RT) {
      const int o = r * nm + (int)m;
      const double *tt = row_entries<BW>(a.tt, r);
      const double *x = pl + first_col<BW>(r, n) * kTile + k;
      auto scalar = [&](int plane, int field, int store, int hline, double visc) {
        const double2 h = s == 3 ? z2(0.0, 0.0) : h_of(hline, o);
        double2 f = z2(0.0, 0.0), d2 = f;
#pragma unroll
        for (int j = 0; j <= 2 * BW; ++j) {
          const double u = x[plane * ps + j * kTile], w = x[(plane + 1) * ps + j * kTile];
          f.x += tt[3 * j] * u;
          f.y += tt[3 * j] * w;
          d2.x += tt[3 * j + 2] * u;
          d2.y += tt[3 * j + 2] * w;
        }
        a.S[field][o] = f;
        a.RK[store][o] = store_new(h, f, d2, visc);
      };
      scalar(P_T, 3, 2, H_HT, visc_t);
      if constexpr (NS == 2) scalar(P_T2, 4, 3, H_HT2, visc_t2);
    }
  __syncthreads();

  // ---- v's right-hand sides: phi_p with the wall velocities at rows 0 and n-1, phi_h with zero there.
  // Opposition control, the extension at the wall rows of the v solve (solve_v_f.f90:251-257,
  // whose commented lines read vold): v at the walls = A * gain * v(+-y_d).  vold is field 10,
  // v after the physical round trip (dft_x_realspace.f90:123), which has no kz Nyquist mode
  // and, at kx = 0, only the Hermitian part (v(kz) + conj v(-kz)) / 2.
  for (int r = rt; r < n; r += RT) {
    double2 p = z2(0.0, 0.0);
    double ph = 0.0;
    if (r > 0 && r < n - 1) {
      const double *tt = row_entries<BW>(a.tt, r);
      const double *x = pl + first_col<BW>(r, n) * kTile + k;
#pragma unroll
      for (int j = 0; j <= 2 * BW; ++j) {
        p.x += tt[3 * j] * x[P_PHI * ps + j * kTile];
        p.y += tt[3 * j] * x[(P_PHI + 1) * ps + j * kTile];
        ph += tt[3 * j] * x[P_PHIH * ps + j * kTile];
      }
    } else if (a.control_amp != 0.0 && live) {
      const int mi = (int)m, kzi = mi / a.nxh, kxi = mi - kzi * a.nxh;
      const double2 *w = a.vwall + (r == 0 ? 0 : nm);
      if (kzi != a.nz / 2) {
        p = w[mi];
        if (kxi == 0) {
          const double2 q = w[(int64_t)((a.nz - kzi) % a.nz) * a.nxh];
          p = z2(0.5 * (p.x + q.x), 0.5 * (p.y - q.y));
        }
        p = zscale(a.control_amp * (double)__ldg(a.gains + mi), p);
      }
    }
    double *y = pl + r * kTile + k;
    y[0] = p.x;
    y[ps] = p.y;
    y[P_VH * ps] = ph;
  }
  __syncthreads();
  if (tid < CT) {
    const bool active = chain < 3;
    sweeps(chain == 2 ? P_VH : active ? chain : 0, NOP, 0, active);
  } else if (producer) {
    feed(2 * C);
  }
  if (__syncthreads_or(!ok)) {
    leave();
    return;
  }

  // ---- the operator rows of the row pairs (r, n-1-r) of a pass go through the ring's memory, which the
  // chains are done with: from L1 a warp's 8 different rows cost 8 cycles a load there, from shared
  // memory 2
  constexpr int RD = op_row_stride(BW);
  const int pairs = (n + 1) / 2, per = min(RT, S * L::slot / (2 * RD));
  double *tlo = ring, *thi = ring + per * RD;  // rows [p0, p0 + pn) and [n - p0 - pn, n - p0)
  auto stage_rows = [&](int p0) {
    const int pn = min(per, pairs - p0);
    const unsigned bytes = (unsigned)(pn * RD * sizeof(double));
    mbar_expect_tx(rowb, 2 * bytes);
    bulk_load(tlo, a.tt + (int64_t)p0 * RD, bytes, rowb);
    bulk_load(thi, a.tt + (int64_t)(n - p0 - pn) * RD, bytes, rowb);
  };
  if (tid == kHelmThreads - 32) stage_rows(0);

  // ---- C1, C2 (solve_v_f.f90:293-298), times (1 + i): the homogeneous derivative is dv_h (1 + i)
  if (tid < kTile) {
    double d[2][3];
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      const int r = w == 0 ? 0 : n - 1;
      const double *tt = row_entries<BW>(a.tt, r), *x = pl + first_col<BW>(r, n) * kTile + tid;
      d[w][0] = d[w][1] = d[w][2] = 0.0;
#pragma unroll
      for (int j = 0; j <= 2 * BW; ++j) {
        const double e1 = tt[3 * j + 1];
        d[w][0] += e1 * x[j * kTile];
        d[w][1] += e1 * x[ps + j * kTile];
        d[w][2] += e1 * x[P_VH * ps + j * kTile];
      }
    }
    const double2 h1 = z2(d[0][2], d[0][2]), hn = z2(d[1][2], d[1][2]);
    const double2 d1 = z2(d[0][0], d[0][1]), dn = z2(d[1][0], d[1][1]);
    const double2 den = zsub(zmul(h1, h1), zmul(hn, hn));
    const double2 C1 = zdiv(zsub(zmul(hn, dn), zmul(h1, d1)), den);
    const double2 C2 = zdiv(zsub(zmul(h1, dn), zmul(hn, d1)), den);
    cc[tid] = C1.x - C1.y;
    cc[kTile + tid] = C1.x + C1.y;
    cc[2 * kTile + tid] = C2.x - C2.y;
    cc[3 * kTile + tid] = C2.x + C2.y;
  }
  __syncthreads();

  // ---- rows r and n-1-r together: each needs the unit-wall solutions of both
  const double2 C1 = z2(cc[k], cc[kTile + k]), C2 = z2(cc[2 * kTile + k], cc[3 * kTile + k]);
  const double alpha = a1n * nu, cd = 1.0 - alpha * k2;
  const double kxk = kk.kx / k2, kzk = kk.kz / k2;
  for (int p0 = 0; p0 < pairs; p0 += per) {
    const int pn = min(per, pairs - p0), r0 = min(p0 + rt, pairs - 1);
    const int o[2] = {r0 * nm + ml, (n - 1 - r0) * nm + ml};
    double2 hv[2], hg[2];  // the nonlinear terms, on their way while the operator rows arrive
    {
      PT q[2][2];
#pragma unroll
      for (int w = 0; w < 2; ++w)
        if (s != 3) {
          q[w][0] = ld_stream(hp(H_HV0) + o[w]);
          q[w][1] = ld_stream(hp(H_G2) + o[w]);
        }
      ok = mbar_wait_bounded(rowb, (p0 / per) & 1);
#pragma unroll
      for (int w = 0; w < 2; ++w) {
        auto wide = [&](int i) { return z2((double)q[w][i].x, (double)q[w][i].y); };
        hv[w] = s == 3 ? z2(0.0, 0.0) : wide(0);
        hg[w] = s == 3 ? z2(0.0, 0.0) : wide(1);
      }
    }
    if (__syncthreads_or(!ok)) {
      leave();
      return;
    }
    if (rt < pn && live) {
      const bool middle = r0 == n - 1 - r0;
      const double *t[2] = {tlo + rt * RD, thi + (pn - 1 - rt) * RD};
      const double *x[2] = {pl + first_col<BW>(r0, n) * kTile + k, pl + first_col<BW>(n - 1 - r0, n) * kTile + k};
      double2 dv[2];
      {  // v and dv/dy
        double2 v[2];
        double vh[2], dvh[2];
#pragma unroll
        for (int w = 0; w < 2; ++w) {
          v[w] = dv[w] = z2(0.0, 0.0);
          vh[w] = dvh[w] = 0.0;
#pragma unroll
          for (int j = 0; j <= 2 * BW; ++j) {
            const double e0 = t[w][3 * j], e1 = t[w][3 * j + 1], *y = x[w] + j * kTile;
            const double re = y[P_T * ps], im = y[(P_T + 1) * ps], h = y[P_VH * ps];
            v[w].x += e0 * re;
            v[w].y += e0 * im;
            dv[w].x += e1 * re;
            dv[w].y += e1 * im;
            vh[w] += e0 * h;
            dvh[w] += e1 * h;
          }
        }
#pragma unroll
        for (int w = 0; w < 2; ++w) {
          if (w == 0 || !middle) a.S[1][o[w]] = zadd(zadd(v[w], zscale(vh[w], C1)), zscale(vh[1 - w], C2));
          dv[w] = zsub(zadd(dv[w], zscale(dvh[w], C1)), zscale(dvh[1 - w], C2));
        }
      }
#pragma unroll
      for (int w = 0; w < 2; ++w) {  // g, u and w
        double2 g = z2(0.0, 0.0), d2g = g;
#pragma unroll
        for (int j = 0; j <= 2 * BW; ++j) {
          const double e0 = t[w][3 * j], e2 = t[w][3 * j + 2], *y = x[w] + j * kTile;
          const double re = y[P_G * ps], im = y[(P_G + 1) * ps];
          g.x += e0 * re;
          g.y += e0 * im;
          d2g.x += e2 * re;
          d2g.y += e2 * im;
        }
        if (w == 0 || !middle) {
          a.RK[0][o[w]] = store_new(hg[w], g, d2g, nu);
          a.S[0][o[w]] = z2(kzk * g.y - kxk * dv[w].y, kxk * dv[w].x - kzk * g.x);  // solve_u_w.f90:27-38
          a.S[2][o[w]] = z2(-kxk * g.y - kzk * dv[w].y, kxk * g.x + kzk * dv[w].x);
        }
      }
      double2 sp[2];  // phi_p's store, and with the unit-wall part (1 - alpha' k2) phi_h + alpha' D2 phi_h
      double ph[2];
#pragma unroll
      for (int w = 0; w < 2; ++w) {
        double2 f = z2(0.0, 0.0), d2f = f;
        double f_h = 0.0, d2f_h = 0.0;
#pragma unroll
        for (int j = 0; j <= 2 * BW; ++j) {
          const double e0 = t[w][3 * j], e2 = t[w][3 * j + 2], *y = x[w] + j * kTile;
          const double re = y[P_PHI * ps], im = y[(P_PHI + 1) * ps], hf = y[P_PHIH * ps];
          f.x += e0 * re;
          f.y += e0 * im;
          d2f.x += e2 * re;
          d2f.y += e2 * im;
          f_h += e0 * hf;
          d2f_h += e2 * hf;
        }
        sp[w] = store_new(hv[w], f, d2f, nu);
        ph[w] = cd * f_h + alpha * d2f_h;
      }
#pragma unroll
      for (int w = 0; w < 2; ++w)
        if (w == 0 || !middle) a.RK[1][o[w]] = zadd(zadd(sp[w], zscale(ph[w], C1)), zscale(ph[1 - w], C2));
    }
    __syncthreads();
    if (tid == kHelmThreads - 32 && p0 + per < pairs) stage_rows(p0 + per);
  }
}

// ------------------------------------------------------------------------------------------
// k_line_hvhg: hvhg.f90:56-159 for a tile of modes, the lines in shared memory as in k_lines (the D0
// factor is the same for all modes and read through L1):
//   h_v = i k2 (kx f2 + kz f4) + D1 c(a3) + D2 c(i kz f4 + i kx f2),  a3 = -kx^2 f1 - 2 kx kz f5 - kz^2 f3
//   h_g = kx kz (f1 - f3) + (kz^2 - kx^2) f5 + D1 c(i kx f4 - i kz f2)
//   h_theta = -(i kx f7 + i kz f9 + D1 c(f8)), with c(f) = D0^{-1} f.
// At substep 1 also D2 D0^{-1} of the RK stores, and the control probes v(+-y_d) = w . v of the
// substep's starting v.  64x65x64 FP64: 38 us against 78 with k_hvhg (wavespace_split.cu), 16x33x16 23 against
// 38, 128x97x128 150 against 132, where k_lines makes up for it.
struct HvhgArgs {
  int n, nxh, nz, substep, nmodes;
  const void *P[11];
  const double2 *RK[4], *v;
  void *hl[H_COUNT];
  const double *l0, *u0, *tt, *wlo, *whi;
  double2 *vwall;
  double control_amp, lmfxr, lmfzr;
  DevScalars *dsc;
};

template <typename PT> __device__ __forceinline__ PT narrow(double2 v);
template <> __device__ __forceinline__ double2 narrow<double2>(double2 v) { return v; }
template <> __device__ __forceinline__ float2 narrow<float2>(double2 v) { return make_float2((float)v.x, (float)v.y); }

template <int BW, typename PT, int NS>
__global__ void __launch_bounds__(kHelmThreads, 3) k_line_hvhg(HvhgArgs a) {
  extern __shared__ __align__(16) double hvhg_lines[];
  if (block_failed(a.dsc)) return;
  constexpr int RT = kHelmThreads / kTile;
  const int n = a.n, s = a.substep, tid = threadIdx.x, nm = a.nmodes, ps = (n | 1) * kTile;
  const int k = tid % kTile, rt = tid / kTile, m = blockIdx.x * kTile + k;
  const bool live = m > 0 && m < nm;
  const int ml = live ? m : 0;
  const ModeK kk = mode_k(ml, a.nxh, a.nz, a.lmfxr, a.lmfzr);
  const double kx = kk.kx, kz = kk.kz, k2 = kk.k2;
  double *pl = hvhg_lines;
  auto prod = [&](int i, int o) {
    const PT v = ld_stream(reinterpret_cast<const PT *>(a.P[i]) + o);
    return z2((double)v.x, (double)v.y);
  };
  auto put = [&](int plane, int r, double2 v) {
    pl[plane * ps + r * kTile + k] = v.x;
    pl[(plane + 1) * ps + r * kTile + k] = v.y;
  };
#pragma unroll 2
  for (int r = rt; r < n; r += RT) {
    const int o = r * nm + ml;
    const double2 f1 = prod(0, o), f2 = prod(1, o), f3 = prod(2, o), f4 = prod(3, o), f5 = prod(4, o);
    put(0, r, zsub(zsub(zscale(-kx * kx, f1), zscale(2.0 * kx * kz, f5)), zscale(kz * kz, f3)));
    put(2, r, prod(6, o));
    put(4, r, z2(kz * f2.y - kx * f4.y, kx * f4.x - kz * f2.x));
    put(6, r, z2(-kz * f4.y - kx * f2.y, kz * f4.x + kx * f2.x));
    if constexpr (NS == 2) put(8, r, prod(9, o));
  }
  __syncthreads();
  // c = D0^{-1} of the first `planes` planes, in place, a thread per plane and mode
  auto solve = [&](int planes) {
    if (rt < planes) {
      double *x = pl + rt * ps + k;
      const double *l0 = a.l0, *u0 = a.u0;
      fixed_fwd<BW, kTile>(x, n, [&](int r, int d) { return l0[r * (2 * BW + 1) + d] * l0[r * (2 * BW + 1)]; },
                           [&](int r) { return l0[r * (2 * BW + 1)]; });
      fixed_bwd<BW, kTile>(x, n, [&](int r, int e) { return u0[r * 2 * BW + e - 1]; });
    }
    __syncthreads();
  };
  // row r of D_d times the coefficients of a plane pair
  auto dot = [&](const double *tt, int d, int plane, int r) {
    const double *x = pl + plane * ps + first_col<BW>(r, n) * kTile + k;
    double2 acc = z2(0.0, 0.0);
#pragma unroll
    for (int j = 0; j <= 2 * BW; ++j) {
      const double e = tt[3 * j + d];
      acc.x += e * x[j * kTile];
      acc.y += e * x[ps + j * kTile];
    }
    return acc;
  };
  solve(NS == 2 ? 10 : 8);
  for (int r = rt; r < n; r += RT) {
    const int o = r * nm + ml;
    const double *tt = row_entries<BW>(a.tt, r);
    const double2 f1 = prod(0, o), f2 = prod(1, o), f3 = prod(2, o), f4 = prod(3, o), f5 = prod(4, o);
    const double2 f7 = prod(5, o), f9 = prod(7, o);
    const double2 hv = zadd(z2(-k2 * (kx * f2.y + kz * f4.y), k2 * (kx * f2.x + kz * f4.x)),
                            zadd(dot(tt, 1, 0, r), dot(tt, 2, 6, r)));
    const double2 hg = zadd(zadd(zscale(kx * kz, zsub(f1, f3)), zscale(kz * kz - kx * kx, f5)), dot(tt, 1, 4, r));
    const double2 t8 = dot(tt, 1, 2, r);
    if (live) {
      reinterpret_cast<PT *>(a.hl[H_HV0])[o] = narrow<PT>(hv);
      reinterpret_cast<PT *>(a.hl[H_G2])[o] = narrow<PT>(hg);
      reinterpret_cast<PT *>(a.hl[H_HT])[o] =
          narrow<PT>(z2(kx * f7.y + kz * f9.y - t8.x, -(kx * f7.x + kz * f9.x + t8.y)));
    }
    if constexpr (NS == 2) {
      const double2 p = prod(8, o), q = prod(10, o), t = dot(tt, 1, 8, r);
      if (live)
        reinterpret_cast<PT *>(a.hl[H_HT2])[o] = narrow<PT>(z2(kx * p.y + kz * q.y - t.x, -(kx * p.x + kz * q.x + t.y)));
    }
  }
  if (s == 1) {
    __syncthreads();
    constexpr int NST = 2 + NS, store_of[4] = {1, 2, 0, 3}, line_of[4] = {H_DP, H_DT, H_DG, H_DT2};
    for (int r = rt; r < n; r += RT)
#pragma unroll
      for (int i = 0; i < NST; ++i) put(2 * i, r, ld_stream(a.RK[store_of[i]] + r * nm + ml));
    __syncthreads();
    solve(2 * NST);
    for (int r = rt; r < n; r += RT) {
      const double *tt = row_entries<BW>(a.tt, r);
#pragma unroll
      for (int i = 0; i < NST; ++i) {
        const double2 d2 = dot(tt, 2, 2 * i, r);
        if (live) reinterpret_cast<double2 *>(a.hl[line_of[i]])[r * nm + m] = d2;
      }
    }
  }
  if (a.control_amp != 0.0) {  // (uniform) the control probes, summed over rt in order
    double2 lo = z2(0.0, 0.0), hi = lo;
    for (int r = rt; r < n; r += RT) {
      const double2 v = ld_stream(a.v + r * nm + ml);
      lo = zadd(lo, zscale(__ldg(a.wlo + r), v));
      hi = zadd(hi, zscale(__ldg(a.whi + r), v));
    }
    __syncthreads();  // the planes are free
    double *red = pl + tid * 4;
    red[0] = lo.x;
    red[1] = lo.y;
    red[2] = hi.x;
    red[3] = hi.y;
    __syncthreads();
    if (tid < kTile && live) {
      double acc[4] = {0.0, 0.0, 0.0, 0.0};
      for (int q = 0; q < RT; ++q)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i] += pl[(q * kTile + tid) * 4 + i];
      a.vwall[m] = z2(acc[0], acc[1]);
      a.vwall[nm + m] = z2(acc[2], acc[3]);
    }
  }
}

// Ring slots of k_lines: three if that many leave room for kHelmBlocks blocks an SM (or for the one that fits).
template <int BW, int NS>
int line_stages(const Handle &h) {
  using L = HelmSmem<BW, NS>;
  const size_t b2 = L::bytes(h.ny, 2), b3 = L::bytes(h.ny, 3);
  return b3 <= (size_t)h.smem_optin && (kHelmBlocks * (b3 + 1024) <= (size_t)h.smem_sm ||
                                        kHelmBlocks * (b2 + 1024) > (size_t)h.smem_sm) ? 3 : 2;
}

// Shared memory of k_line_hvhg: its planes, and at least the probes' sums.
size_t line_hvhg_bytes(const Handle &h) {
  const size_t planes = (size_t)(h.nsc == 2 ? 10 : 8) * (size_t)(h.ny | 1) * kTile;
  return sizeof(double) * (planes > 4 * kHelmThreads ? planes : 4 * kHelmThreads);
}

int smem_attr(cudaDeviceAttr attr) {
  int dev = 0, v = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&v, attr, dev) != cudaSuccess) return 0;
  return v;
}

HelmArgs helm_args(Handle &h, int substep, const double *dt_ptr) {
  HelmArgs a{};
  const OpsOffsets off = ops_offsets(h.bw, h.ny);
  a.n = h.ny;
  a.nxh = h.nxh;
  a.nz = h.nz;
  a.substep = substep;
  a.nmodes = h.nmodes;
  a.ns = h.ns;
  for (int f = 0; f < 3 + h.nsc; ++f) a.S[f] = h.S + f * h.ns;
  for (int f = 0; f < 2 + h.nsc; ++f) a.RK[f] = h.RK + f * h.ns;
  for (int i = 0; i < H_COUNT; ++i) {
    const bool prod = i <= H_V3 || i == H_HT2;  // at the products' type
    a.hl[i] = prod && h.mixed ? (const void *)(reinterpret_cast<const float2 *>(h.ec) + i * h.ns) : h.ec + i * h.ns;
  }
  a.tabs = h.dops + off.t0;
  a.tt = h.dops + off.tt;
  a.vwall = h.vwall;
  a.gains = h.gains;
  a.control_amp = h.cfg.control_amp;
  a.nu = h.cfg.nu;
  a.pr = h.cfg.pr;
  a.pr2 = h.cfg.pr2;
  a.lmfxr = h.lmfxr;
  a.lmfzr = h.lmfzr;
  a.dsc = h.dsc;
  a.dt_ptr = dt_ptr ? dt_ptr : &h.dsc->dt;
  a.vf = h.lvf;
  // one factor set per operator; with the factor cache (a fixed time step) per substep too
  const int64_t set = tile_factor_doubles(h);
  const int nop = 1 + h.nsc;
  const int at = h.fcdt ? nop * (substep - 1) : 0;
  for (int o = 0; o < nop; ++o) a.fac[o] = h.lf + (at + o) * set;
  a.fcdt = h.fcdt ? h.fcdt + (substep - 1) : nullptr;
  a.fcount = h.fcount ? h.fcount + (substep - 1) : nullptr;
  a.cached = h.fcdt && h.tune.fcache;
  return a;
}

template <int BW>
cudaError_t helm_bw(Handle &h, int substep, const double *dt_ptr, cudaStream_t st) {
  const HelmArgs a = helm_args(h, substep, dt_ptr);
  const unsigned tiles = (unsigned)((h.nmodes + kTile - 1) / kTile);
  auto go = [&]<typename PT, int NS>() {
    HelmArgs b = a;
    b.stages = line_stages<BW, NS>(h);
    k_lines<BW, PT, NS><<<tiles, kHelmThreads, HelmSmem<BW, NS>::bytes(h.ny, b.stages), st>>>(b);
  };
  if (h.mixed) h.nsc == 2 ? go.template operator()<float2, 2>() : go.template operator()<float2, 1>();
  else h.nsc == 2 ? go.template operator()<double2, 2>() : go.template operator()<double2, 1>();
  return cudaGetLastError();
}

template <int BW>
cudaError_t hvhg_bw(Handle &h, int substep, cudaStream_t st) {
  const OpsOffsets off = ops_offsets(h.bw, h.ny);
  HvhgArgs a{};
  a.n = h.ny;
  a.nxh = h.nxh;
  a.nz = h.nz;
  a.substep = substep;
  a.nmodes = (int)h.nmodes;
  for (int i = 0; i < 5 + 3 * h.nsc; ++i)
    a.P[i] = h.mixed ? (const void *)(reinterpret_cast<const float2 *>(h.P) + i * h.ns)
                     : reinterpret_cast<const double2 *>(h.P) + i * h.ns;
  const HelmArgs l = helm_args(h, substep, nullptr);
  for (int i = 0; i < 4; ++i) a.RK[i] = l.RK[i];
  a.v = l.S[1];
  for (int i = 0; i < H_COUNT; ++i) a.hl[i] = const_cast<void *>(l.hl[i]);
  const int64_t tw = (int64_t)h.ny * (4 * BW + 1);
  a.l0 = h.dops + off.t0 + 3 * tw;
  a.u0 = a.l0 + (int64_t)h.ny * (2 * BW + 1);
  a.tt = h.dops + off.tt;
  a.wlo = h.dops + off.wlo;
  a.whi = h.dops + off.whi;
  a.vwall = h.vwall;
  a.control_amp = h.cfg.control_amp;
  a.lmfxr = h.lmfxr;
  a.lmfzr = h.lmfzr;
  a.dsc = h.dsc;
  const unsigned tiles = (unsigned)((h.nmodes + kTile - 1) / kTile);
  const size_t bytes = line_hvhg_bytes(h);
  if (h.mixed && h.nsc == 2) k_line_hvhg<BW, float2, 2><<<tiles, kHelmThreads, bytes, st>>>(a);
  else if (h.mixed) k_line_hvhg<BW, float2, 1><<<tiles, kHelmThreads, bytes, st>>>(a);
  else if (h.nsc == 2) k_line_hvhg<BW, double2, 2><<<tiles, kHelmThreads, bytes, st>>>(a);
  else k_line_hvhg<BW, double2, 1><<<tiles, kHelmThreads, bytes, st>>>(a);
  return cudaGetLastError();
}

template <int BW>
cudaError_t factor_bw(Handle &h, int substep, const double *dt_ptr, cudaStream_t st) {
  const HelmArgs a = helm_args(h, substep, dt_ptr);
  k_line_factor<BW><<<dim3((unsigned)((h.nmodes + 31) / 32), (unsigned)(1 + h.nsc)), 32, 0, st>>>(a);
  return cudaGetLastError();
}

template <int BW>
cudaError_t prepare_bw(Handle &h, cudaStream_t st) {
  auto lim = [&](auto kern) {
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, h.smem_optin);
  };
  cudaError_t e = lim(k_lines<BW, float2, 1>);
  if (e == cudaSuccess) e = lim(k_lines<BW, double2, 1>);
  if (e == cudaSuccess) e = lim(k_line_hvhg<BW, float2, 1>);
  if (e == cudaSuccess) e = lim(k_line_hvhg<BW, double2, 1>);
  if (e == cudaSuccess) e = lim(k_line_hvhg<BW, float2, 2>);
  if (e == cudaSuccess) e = lim(k_line_hvhg<BW, double2, 2>);
  if (e == cudaSuccess) e = lim(k_lines<BW, float2, 2>);
  if (e == cudaSuccess) e = lim(k_lines<BW, double2, 2>);
  if (e != cudaSuccess) return e;
  HelmArgs a = helm_args(h, 1, nullptr);
  a.fac[0] = nullptr;  // v's operator
  k_line_factor<BW><<<dim3((unsigned)((h.nmodes + 31) / 32)), 32, 0, st>>>(a);
  return cudaGetLastError();
}

template <typename F> auto with_bw(int bw, F &&f) {
  switch (bw) {
    case 2: return f.template operator()<2>();
    case 3: return f.template operator()<3>();
    case 4: return f.template operator()<4>();
    case 5: return f.template operator()<5>();
    case 6: return f.template operator()<6>();
    case 7: return f.template operator()<7>();
    default: return cudaErrorInvalidValue;
  }
}

// Whether two blocks of k_lines are resident on an SM.
bool two_lines(const Handle &h) {
  bool two = false;
  with_bw(h.bw, [&]<int BW>() {
    const size_t bytes = h.nsc == 2 ? HelmSmem<BW, 2>::bytes(h.ny, line_stages<BW, 2>(h))
                                    : HelmSmem<BW, 1>::bytes(h.ny, line_stages<BW, 1>(h));
    two = kHelmBlocks * (bytes + 1024) <= (size_t)h.smem_sm;
    return cudaSuccess;
  });
  return two;
}

// Up to how many modes the line solver is the faster one, from whole steps with either solver (ratio line
// solver / sweeps, FP64 and mixed, ny from 33 to 353, 4096 to 15360 modes; below 4096 it is 0.25 to 0.9
// everywhere).  With more modes the sweeps have the warps to hide their latency; the line solver loses
// residency with ny, k_line_hvhg's second block an SM above all (its planes: ny = 227 with one scalar, 181
// with two), and so does its lead.  Sweeps that have to factor each substep (a CFL time step, two
// scalars) lose more the wider the band.
int64_t line_modes(const Handle &h) {
  const int bw = h.bw;
  const bool cached = factor_cache_possible(h);
  const bool two_hvhg = 2 * (line_hvhg_bytes(h) + 1024) <= (size_t)h.smem_sm;
  constexpr int64_t all = 12000;  // (12800 modes at band width 4: 0.95 to 1.07)
  if (!cached && bw >= 6) return all;  // 0.43 to 1.00 up to 13824 modes, also with one block an SM
  if (!two_hvhg) {
    if (cached) return bw <= 4 ? 8700   // 8192 modes 0.92 to 0.98, 9216 0.97 to 1.05
                       : 7000;          // 6144 modes 0.91 to 0.98, 8192 1.00 to 1.08
    if (h.nsc == 2) return bw == 4 ? 6000   // 5120 modes 0.90 to 0.95, 6144 0.99 to 1.04
                           : 7000;          // 6144 modes 0.94 to 0.98, 8192 1.03 to 1.06
    return bw <= 4 ? 7000   // 6144 modes 0.92 to 0.97, 8192 1.01 to 1.04
           : 8700;          // 8192 modes 0.93, 9216 1.00
  }
  if (cached) {
    if (bw <= 4) return h.ny < 48 ? 10900 : all;  // 11520 modes 0.92 to 0.98, at ny = 33 0.99 to 1.03
    if (h.ny < 48) return 7000;                   // 6144 modes 0.88, 8192 1.03 to 1.05
    return bw == 5 ? 10900   // 10368 modes 0.92 to 1.01, 11520 0.98 to 1.05
           : 9000;           // 8192 modes 0.93 to 1.03, 9216 0.97 to 1.07
  }
  if (h.nsc == 2) {
    // 11520 modes 0.95 to 1.00 (ny = 33: 10240 0.98 to 1.02); with one block of k_lines an SM 6144 modes 0.86
    // to 0.93 and 8192 0.98 to 1.03, at band width 5 11520 modes 0.97 to 1.02
    if (bw == 5) return all;
    if (!two_lines(h)) return 7600;
    return h.ny < 48 ? 10000 : all;
  }
  if (bw <= 3) {
    if (h.ny < 48) return 7000;          // 6144 modes 0.86 to 0.95, 8192 1.03 to 1.06
    if (!two_lines(h)) return 8700;      // 8192 modes 0.96 to 1.03, 9216 0.99 to 1.05
    return h.ny < 96 ? 11000 : all;      // at ny = 65 10368 modes 0.99 to 1.01, 11520 1.02 to 1.04
  }
  return h.ny < 48 && bw == 4 ? 10900 : all;  // 11520 modes 0.95 to 1.02, at ny = 33 1.01 to 1.02
}

}  // namespace

bool line_solver_fits(Handle &h) {
  h.smem_optin = smem_attr(cudaDevAttrMaxSharedMemoryPerBlockOptin);
  h.smem_sm = smem_attr(cudaDevAttrMaxSharedMemoryPerMultiprocessor);
  size_t bytes = (size_t)-1;
  with_bw(h.bw, [&]<int BW>() {
    bytes = h.nsc == 2 ? HelmSmem<BW, 2>::bytes(h.ny, 2) : HelmSmem<BW, 1>::bytes(h.ny, 2);
    return cudaSuccess;
  });
  return bytes <= (size_t)h.smem_optin;
}

bool line_solver_pays(const Handle &h) { return h.nmodes <= line_modes(h); }

int64_t tile_factor_doubles(const Handle &h) {
  const int64_t tiles = (h.nmodes + kTile - 1) / kTile, bw = h.bw;
  return tiles * kTile * ((int64_t)h.ny * (2 * bw + 1) + 2 * bw * (bw + 1));  // TileFac::size
}

cudaError_t prepare_line_solver(Handle &h, cudaStream_t st) {
  return with_bw(h.bw, [&]<int BW>() { return prepare_bw<BW>(h, st); });
}

cudaError_t launch_line_hvhg(Handle &h, int substep, cudaStream_t st) {
  return with_bw(h.bw, [&]<int BW>() { return hvhg_bw<BW>(h, substep, st); });
}

cudaError_t launch_line_factor(Handle &h, int substep, const double *dt_ptr, cudaStream_t st) {
  return with_bw(h.bw, [&]<int BW>() { return factor_bw<BW>(h, substep, dt_ptr, st); });
}

cudaError_t launch_line_solver(Handle &h, int substep, const double *dt_ptr, cudaStream_t st) {
  return with_bw(h.bw, [&]<int BW>() { return helm_bw<BW>(h, substep, dt_ptr, st); });
}

}  // namespace kmm
