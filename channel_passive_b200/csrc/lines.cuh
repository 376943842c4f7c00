// lines.cuh - per-mode wall-normal solves on lines held in shared memory.
//
// A block owns a tile of kTile modes.  The lines of the tile's solves lie in shared memory as
// real planes [row][mode] (real and imaginary parts apart), because the operators are real: every
// real chain of every solve is a thread of its own.  The serial part, a forward and a backward
// substitution in place, is all such a thread does; the band products (D0, D1, D2 times the
// coefficients) that follow run over all rows and modes in parallel.  One thread that did both for a
// row, staged a row ahead from global memory, took 700 to 1500 cycles a row, most of it latency.
//
// The LU factors of an operator are kept tile by tile (TileFac), so that the kChunk rows of a tile
// that a sweep needs next are one contiguous run, fetched by one cp.async.bulk into a ring of slots
// ahead of the chains.  Rows are 0-based here.
#pragma once

#include <cuda_runtime.h>

#include "kmm_internal.h"
#include "sweeps.cuh"
#include "tma.cuh"

namespace kmm {

constexpr int kTile = kTileModes;  // modes of a block
constexpr int kChunk = 24;         // rows of one staged copy
constexpr int kMaxStages = 3;      // ring slots, where shared memory has room for them

// One operator's factors of one tile, in doubles, each entry for kTile modes next to each other (in
// fwd and bwd two entries of a mode are neighbours, for 16-byte loads: entry_at), in the order the
// chains use them (by columns: what the solution of a row adds to the rows that follow):
//   fwd  [n][BW+1]  row r: 1 / L(r+BW, r+BW), then l(r+k, r) = L(r+k, r) / L(r+k, r+k) for k = 1..BW
//   fx   [BW][BW]   l(r, r-d) for d = BW+1..2BW of the last BW rows r (the only ones that reach there)
//   rp   [BW]       1 / L(r, r) of the first BW rows
//   bwd  [n][BW]    row r: U(r-k, r), k = 1..BW (unit diagonal)
//   bx   [BW][BW]   U(r, r+e) for e = BW+1..2BW of the first BW rows r
// L is kept divided by its pivot so that z_r = b_r / L(r, r) - sum_d l(r, d) z_{r-d} hangs on z_{r-1}
// by one multiply-add.  Entries that name rows outside the matrix are not written and not used.
template <int BW>
struct TileFac {
  static __host__ __device__ constexpr int64_t fx(int n) { return (int64_t)kTile * n * (BW + 1); }
  static __host__ __device__ constexpr int64_t bwd(int n) { return fx(n) + ext; }
  static __host__ __device__ constexpr int64_t bx(int n) { return bwd(n) + (int64_t)kTile * n * BW; }
  static __host__ __device__ constexpr int64_t size(int n) { return bx(n) + ext; }
  // doubles of the fx + rp block, and of the bx block (padded to the same)
  static constexpr int ext = kTile * BW * (BW + 1);
};

// Where entry k of a row of W entries lies for mode m of the tile.
__host__ __device__ constexpr int entry_at(int W, int k, int m) {
  return k < W / 2 * 2 ? (k / 2 * kTile + m) * 2 + k % 2 : k * kTile + m;
}

// U of one mode inside its tile's TileFac, for LuSweep (1-based rows); b the tile's bwd, x the mode's bx.
template <int BW>
struct TileU {
  double *b, *x;
  int n, m;
  __device__ __forceinline__ double get(int r, int e) const {
    if (e <= BW) return r + e <= n ? b[(r + e - 1) * BW * kTile + entry_at(BW, e - 1, m)] : 0.0;
    return r <= BW ? x[((r - 1) * BW + e - BW - 1) * kTile] : 0.0;
  }
  __device__ __forceinline__ void set(int r, int e, double v) const {
    if (e <= BW) {
      if (r + e <= n) b[(r + e - 1) * BW * kTile + entry_at(BW, e - 1, m)] = v;
    } else if (r <= BW) {
      x[((r - 1) * BW + e - BW - 1) * kTile] = v;
    }
  }
};

// Rows of a slot of the ring: a sweep's last chunk also takes the last BW rows (chunk_rows).
template <int BW> constexpr int slot_rows() { return kChunk + BW; }
// Chunks of a sweep: the rows before the last BW in runs of kChunk, the last BW with the last run.
template <int BW> __device__ __forceinline__ int sweep_chunks(int n) { return (n - BW + kChunk - 1) / kChunk; }
__device__ __forceinline__ int chunk_rows(int c, int C, int n) { return c + 1 < C ? kChunk : n - c * kChunk; }

// Shared-memory accesses that keep a batch's loads together, ahead of its arithmetic (p a byte address,
// i doubles on).
__device__ __forceinline__ double lds(unsigned p, int i) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(p + 8u * (unsigned)i) : "memory");
  return v;
}
__device__ __forceinline__ void sts(unsigned p, int i, double v) {
  asm volatile("st.shared.f64 [%0], %1;" ::"r"(p + 8u * (unsigned)i), "d"(v) : "memory");
}

// Rows whose inputs a chain loads together: their shared-memory latency is paid once a batch.
template <int BW> constexpr int chain_batch() { return BW <= 5 ? 4 : 2; }

// The W staged entries of one row: co the row's first double, m the mode (LDS.128 for each pair).
template <int W>
__device__ __forceinline__ void load_entries(double (&l)[W], unsigned co, int m) {
#pragma unroll
  for (int k = 0; k + 1 < W; k += 2)
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];"
                 : "=d"(l[k]), "=d"(l[k + 1])
                 : "r"(co + 8u * (unsigned)entry_at(W, k, m))
                 : "memory");
  if constexpr (W % 2 == 1)
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(l[W - 1]) : "r"(co + 8u * (unsigned)entry_at(W, W - 1, m)) : "memory");
}

// The chains are right-looking: once z_r is known it goes into the sums of the BW rows that follow, so
// that a row costs the latency of one FP64 multiply-add (8 cycles, the one into row r+1; the others
// issue under it) or the issue of its loads, whichever is longer.  Summing row r's BW terms when its
// turn comes took 155 cycles a row (BW = 4).  acc[k] is the sum of row r+k so far.
// The inputs of RB rows are loaded together (46 cycles a row alone on an SM with batches of 4: 12 of
// arithmetic, 15 of load issue, the rest latency; loading a batch ahead of the one at work took 54).
template <int BW, int RB>
struct FwdBatch {
  double b[RB], l[RB][BW + 1];  // l[0]: 1 / L of row r+BW, l[k]: l(r+k, r)
  // x the chain's plane column at row r (row stride kTile), co row r's staged factors, left = n - r
  __device__ __forceinline__ void load(unsigned x, unsigned co, int m, int left) {
#pragma unroll
    for (int i = 0; i < RB; ++i) {
      load_entries<BW + 1>(l[i], co + 8u * i * (BW + 1) * kTile, m);
      b[i] = lds(x, min(i + BW, left - 1) * kTile);  // (a row past the last is not used)
    }
  }
  __device__ __forceinline__ void run(unsigned x, double (&acc)[BW]) const {
    double z[RB];
#pragma unroll
    for (int i = 0; i < RB; ++i) {
      z[i] = acc[0];
#pragma unroll
      for (int k = 1; k < BW; ++k) acc[k - 1] = acc[k] - l[i][k] * z[i];
      acc[BW - 1] = b[i] * l[i][0] - l[i][BW] * z[i];
    }
#pragma unroll
    for (int i = 0; i < RB; ++i) sts(x, i * kTile, z[i]);
  }
};

// The same of a backward substitution, descending from row r: acc[k] the sum of row r-k.
template <int BW, int RB>
struct BwdBatch {
  double b[RB], u[RB][BW];  // u[k-1]: U(r-k, r)
  __device__ __forceinline__ void load(unsigned x, unsigned co, int m, int r) {
#pragma unroll
    for (int i = 0; i < RB; ++i) {
      load_entries<BW>(u[i], co - 8u * i * BW * kTile, m);
      b[i] = lds(x, -min(i + BW, r) * kTile);
    }
  }
  __device__ __forceinline__ void run(unsigned x, double (&acc)[BW]) const {
    double z[RB];
#pragma unroll
    for (int i = 0; i < RB; ++i) {
      z[i] = acc[0];
#pragma unroll
      for (int k = 1; k < BW; ++k) acc[k - 1] = acc[k] - u[i][k - 1] * z[i];
      acc[BW - 1] = b[i] - u[i][BW - 1] * z[i];
    }
#pragma unroll
    for (int i = 0; i < RB; ++i) sts(x, -i * kTile, z[i]);
  }
};

// Chunk c (of C) of a forward substitution of the chain whose plane column is x (row 0); co the chunk's
// staged factors, fx TileFac's fx block (of mode m).  n > 2 BW.
template <int BW>
__device__ __forceinline__ void fwd_chunk(unsigned x, unsigned co, unsigned fx, int m, int c, int C, int n,
                                          double (&acc)[BW]) {
  constexpr int RB = chain_batch<BW>();
  constexpr unsigned row = 8u * (BW + 1) * kTile;
  int r = c * kChunk;
  const int r1 = c + 1 < C ? r + kChunk : n - BW;  // the regular rows
  if (c == 0) {
#pragma unroll
    for (int k = 0; k < BW; ++k)
      acc[k] = lds(x, k * kTile) * lds(fx, (BW * BW + k) * kTile);  // rp
  }
  x += 8u * (unsigned)(r * kTile);
#pragma unroll 1
  for (; r + RB <= r1; r += RB) {
    FwdBatch<BW, RB> q;
    q.load(x, co, m, n - r);
    q.run(x, acc);
    co += RB * row;
    x += 8u * (unsigned)(RB * kTile);
  }
#pragma unroll 1
  for (; r < r1; ++r) {
    FwdBatch<BW, 1> q;
    q.load(x, co, m, n - r);
    q.run(x, acc);
    co += row;
    x += 8u * (unsigned)(kTile);
  }
  if (c + 1 == C) {
    // the last BW rows: their entries past the band reach rows before r - 1, all known
#pragma unroll
    for (int k = 0; k < BW; ++k)
#pragma unroll
      for (int d = 2 * BW; d > BW; --d)
        if (k >= d - BW - 1) acc[k] -= lds(fx, (k * BW + d - BW - 1) * kTile) * lds(x, (k - d) * kTile);
    FwdBatch<BW, BW> last;
    last.load(x, co, m, BW);
    last.run(x, acc);
  }
}

// Chunk c (of C) of a backward substitution; bx TileFac's bx block (of mode m).
template <int BW>
__device__ __forceinline__ void bwd_chunk(unsigned x, unsigned co, unsigned bx, int m, int c, int C, int n,
                                          double (&acc)[BW]) {
  constexpr int RB = chain_batch<BW>();
  constexpr unsigned row = 8u * BW * kTile;
  const int r0 = c == 0 ? BW : c * kChunk;  // the regular rows
  int r = c * kChunk + chunk_rows(c, C, n) - 1;
  if (c + 1 == C) {
#pragma unroll
    for (int k = 0; k < BW; ++k) acc[k] = lds(x, (n - 1 - k) * kTile);
  }
  x += 8u * (unsigned)(r * kTile);
  co += (unsigned)(r - c * kChunk) * row;
#pragma unroll 1
  for (; r - RB + 1 >= r0; r -= RB) {
    BwdBatch<BW, RB> q;
    q.load(x, co, m, r);
    q.run(x, acc);
    co -= RB * row;
    x += 8u * (unsigned)(-RB * kTile);
  }
#pragma unroll 1
  for (; r >= r0; --r) {
    BwdBatch<BW, 1> q;
    q.load(x, co, m, r);
    q.run(x, acc);
    co -= row;
    x += 8u * (unsigned)(-kTile);
  }
  if (c == 0) {
    // the first BW rows, from row BW-1 down
#pragma unroll
    for (int k = 0; k < BW; ++k)
#pragma unroll
      for (int e = 2 * BW; e > BW; --e)
        if (k >= e - BW - 1)
          acc[k] -= lds(bx, ((BW - 1 - k) * BW + e - BW - 1) * kTile) * lds(x, (e - k) * kTile);
    BwdBatch<BW, BW> last;
    last.load(x, co, m, BW - 1);
    last.run(x, acc);
  }
}

// Forward substitution in place over n values ST apart, right-looking, the factors shared by all modes: lf(r, d) = L(r, r-d) / L(r, r) for
// d = 1..2BW, rp(r) = 1 / L(r, r).
template <int BW, int ST, typename LF, typename RP>
__device__ __forceinline__ void fixed_fwd(double *x, int n, LF lf, RP rp) {
  constexpr int RB = 4;
  double acc[BW];
#pragma unroll
  for (int k = 0; k < BW; ++k) acc[k] = x[k * ST] * rp(k);
  int r = 0;
  for (; r + RB + BW <= n - BW; r += RB) {
    double b[RB], l[RB][BW], z[RB];
#pragma unroll
    for (int i = 0; i < RB; ++i) {
      b[i] = x[(r + i + BW) * ST] * rp(r + i + BW);
#pragma unroll
      for (int k = 1; k <= BW; ++k) l[i][k - 1] = lf(r + i + k, k);
    }
#pragma unroll
    for (int i = 0; i < RB; ++i) {
      z[i] = acc[0];
#pragma unroll
      for (int k = 1; k < BW; ++k) acc[k - 1] = acc[k] - l[i][k - 1] * z[i];
      acc[BW - 1] = b[i] - l[i][BW - 1] * z[i];
    }
#pragma unroll
    for (int i = 0; i < RB; ++i) x[(r + i) * ST] = z[i];
  }
  for (; r < n; ++r) {  // the rows near the end, which reach 2BW rows back
    double t = x[r * ST] * rp(r);
    for (int d = min(r, r >= n - BW ? 2 * BW : BW); d >= 1; --d) t -= lf(r, d) * x[(r - d) * ST];
    x[r * ST] = t;
  }
}

// Backward substitution: uf(r, e) = U(r, r+e), e = 1..2BW.
template <int BW, int ST, typename UF>
__device__ __forceinline__ void fixed_bwd(double *x, int n, UF uf) {
  constexpr int RB = 4;
  double acc[BW];
#pragma unroll
  for (int k = 0; k < BW; ++k) acc[k] = x[(n - 1 - k) * ST];
  int r = n - 1;
  for (; r - RB - BW + 1 >= BW; r -= RB) {
    double b[RB], u[RB][BW], z[RB];
#pragma unroll
    for (int i = 0; i < RB; ++i) {
      b[i] = x[(r - i - BW) * ST];
#pragma unroll
      for (int k = 1; k <= BW; ++k) u[i][k - 1] = uf(r - i - k, k);
    }
#pragma unroll
    for (int i = 0; i < RB; ++i) {
      z[i] = acc[0];
#pragma unroll
      for (int k = 1; k < BW; ++k) acc[k - 1] = acc[k] - u[i][k - 1] * z[i];
      acc[BW - 1] = b[i] - u[i][BW - 1] * z[i];
    }
#pragma unroll
    for (int i = 0; i < RB; ++i) x[(r - i) * ST] = z[i];
  }
  for (; r >= 0; --r) {
    double t = x[r * ST];
    for (int e = min(n - 1 - r, r < BW ? 2 * BW : BW); e >= 1; --e) t -= uf(r, e) * x[(r + e) * ST];
    x[r * ST] = t;
  }
}

// Whether a failed step is to be left untouched, decided once per block: another block of the same grid, or a
// kernel beside it, may raise the flag while this one starts, and threads that left on their own reading of
// it would leave the others at barriers that were never set up.
__device__ __forceinline__ bool block_failed(const DevScalars *dsc) {
  return __syncthreads_or(threadIdx.x == 0 && dsc->err != 0);
}

// Row r of an operator spans 2BW+1 columns from here (the near-boundary packing of the first and
// last BW rows, LABS_full_to_band, module_labs.f90:301-328).
template <int BW>
__device__ __forceinline__ int first_col(int r, int n) {
  const int s = r - BW;
  return s < 0 ? 0 : s > n - 1 - 2 * BW ? n - 1 - 2 * BW : s;
}
// The operator rows as the mat-vecs read them: row r's 2BW+1 columns, D0, D1, D2 of a column next to
// each other, in op_row_stride(BW) doubles (OpsOffsets::tt).  28 KB at ny = 129 and BW = 4; the offset
// tables (half zeros) are 52 KB.
template <int BW>
__device__ __forceinline__ const double *row_entries(const double *tt, int r) {
  return tt + (int64_t)r * op_row_stride(BW);
}

// Streamed data that must not push the operator rows out of L1.
template <typename T>
__device__ __forceinline__ T ld_stream(const T *p) {
  T v;
  if constexpr (sizeof(T) == 16)
    asm volatile("ld.global.L1::no_allocate.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  else
    asm volatile("ld.global.L1::no_allocate.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
  return v;
}

// Low-storage RK3 coefficients alpha, beta, gamma, zeta of substeps 1-3
// (RK3_initialize, module_runge_kutta.f90:34-45).
static __constant__ double c_rk[4][3] = {{29.0 / 96.0, -3.0 / 40.0, 1.0 / 6.0},
                                         {37.0 / 160.0, 5.0 / 24.0, 1.0 / 6.0},
                                         {8.0 / 15.0, 5.0 / 12.0, 3.0 / 4.0},
                                         {0.0, -17.0 / 60.0, -5.0 / 12.0}};
__device__ __forceinline__ double rkc(int c, int s) { return c_rk[c - 1][s - 1]; }

struct ModeK {
  double kx, kz, k2;
};
__device__ __forceinline__ ModeK mode_k(int mi, int nxh, int nz, double lmfxr, double lmfzr) {
  const int kzi = mi / nxh, kxi = mi - kzi * nxh;
  const int kzint = (kzi <= nz / 2) ? kzi : kzi - nz;  // set_waveno
  ModeK k;
  k.kx = kxi * lmfxr;                                   // wavespace.f90:69
  k.kz = kzint * lmfzr;
  k.k2 = k.kx * k.kx + k.kz * k.kz;
  return k;
}

// A = ca D0 - cb D2 with the Dirichlet first / last rows, as an offset row (|e| <= BW only
// for a centre row, which is never a wall row); 1-based row.
template <int BW>
__device__ __forceinline__ void helm_row(const Tabs<BW> &tb, int r, int n, double ca, double cb, double *out,
                                         bool centre) {
  const double *r0 = trow<BW>(tb.t0, r), *r2 = trow<BW>(tb.t2, r);
  if (centre) {
#pragma unroll
    for (int e = -BW; e <= BW; ++e) out[e + 2 * BW] = ca * r0[e] - cb * r2[e];
    return;
  }
  if (r == 1 || r == n) {
#pragma unroll
    for (int e = -2 * BW; e <= 2 * BW; ++e) out[e + 2 * BW] = 0.0;
    out[2 * BW] = ca * r0[0] - cb * r2[0];
    return;
  }
#pragma unroll
  for (int e = -2 * BW; e <= 2 * BW; ++e) out[e + 2 * BW] = ca * r0[e] - cb * r2[e];
}

// (D2 - k^2 D0) with the wall rows replaced by D0 (v given there), solve_v_f.f90:95-140.
template <int BW>
__device__ __forceinline__ void vrow(const Tabs<BW> &tb, int r, int n, double k2, double *row, bool centre) {
  const double *r0 = trow<BW>(tb.t0, r), *r2 = trow<BW>(tb.t2, r);
  if (centre) {
#pragma unroll
    for (int e = -BW; e <= BW; ++e) row[e + 2 * BW] = -k2 * r0[e] + r2[e];
    return;
  }
  if (r == 1 || r == n) {
#pragma unroll
    for (int e = -2 * BW; e <= 2 * BW; ++e) row[e + 2 * BW] = 0.0;
    row[2 * BW] = r0[0];
    return;
  }
#pragma unroll
  for (int e = -2 * BW; e <= 2 * BW; ++e) row[e + 2 * BW] = -k2 * r0[e] + r2[e];
}

// Lines hvhg hands to the Helmholtz solves.  (The line solver's k_line_hvhg fills H_HV0 with all of h_v
// and H_G2 with all of h_g, and leaves H_V2, H_V3 and H_G3.)
// k_hvhg's:  The six nonlinear-term lines H_HV0..H_V3 are combinations
// of the products and are stored at the products' precision PT (float2 in the mixed path, packed
// at (PT *)hl + i * ns); the substep-1 lines H_DP, H_DT, H_DG (D2 D0^{-1} of the FP64 RK stores)
// stay double2 at hl + i * ns.
// A second passive scalar adds H_HT2 (its nonlinear term, at PT like H_HT) and H_DT2 (substep 1,
// double2 like H_DT).
enum HLine { H_HV0 = 0, H_HT, H_G2, H_V2, H_G3, H_V3, H_DP, H_DT, H_DG, H_HT2, H_DT2, H_COUNT };

template <typename PT> __device__ __forceinline__ double2 ldp(const PT *p);
template <> __device__ __forceinline__ double2 ldp<double2>(const double2 *p) { return *p; }
template <> __device__ __forceinline__ double2 ldp<float2>(const float2 *p) {
  const float2 v = *p;
  return make_double2((double)v.x, (double)v.y);
}

}  // namespace kmm
