/*
 * gp_tiles.cuh -- what the time-step kernels share, generic in the field type R:
 * tile geometry, the boundary copy tables, divisions by the spacings, the FP32
 * rounding, the dc/dmu solve, the progress record's buffers and a simulation's
 * layout.
 *
 * Data layout in HBM: one plane per field (phi_a, mu_k), interior cells only,
 * row x, column y contiguous.  The reference's three ghost layers are never
 * stored: after every boundary copy a ghost cell holds an interior cell, so
 * loads map ghost coordinates through the copy tables (remap) instead.
 */
#pragma once
#include "gp_math.cuh"

namespace gpd {

constexpr int TX = 8;    /* rows per tile    */
constexpr int TY = 32;   /* columns per tile */
constexpr int NT = TX * TY;
constexpr int SW = TY + 2, SH = TX + 2, SS = SW * SH;
constexpr int NXF = (TX + 1) * TY;       /* x-faces of a tile */
constexpr int NYF = TX * (TY + 1);       /* y-faces of a tile */

struct Grid {
  int mx, my;            /* interior size */
  int pitch;             /* row pitch of state planes (elements) */
  long long plane;       /* elements per state plane */
  int dpitch;            /* row pitch of the delta-phi buffer */
  long long dplane;      /* elements per delta-phi plane ((mx+2) rows) */
  int sx0, sx1;          /* rows the progress statistics cover (a slab's own rows; all by default) */
};

/* offset of a cell in its plane (a plane may hold more than 2^31 cells) */
__host__ __device__ __forceinline__ long long plane_offset(const Grid &g, int x, int y) {
  return (long long)x * g.pitch + y;
}

/* rows moved by one gp_rows_pack / gp_rows_unpack call: item i is row
 * row[i] of state field field[i] */
constexpr int ROW_ITEMS_MAX = 64;
struct RowItems {
  int field[ROW_ITEMS_MAX];
  int row[ROW_ITEMS_MAX];
};

/* the cell's row is counted by the progress statistics */
__device__ __forceinline__ bool stat_row(const Grid &g, int x) { return x >= g.sx0 && x < g.sx1; }

/* interior coordinate v in [-3, m+2] -> interior coordinate it is a copy of
 * (assign_buffer_points_conditions / assign_boundary_points_values,
 * utility_functions.h:471-654): Neumann mirrors about the boundary cell,
 * periodic wraps with period m-1. */
__host__ __device__ __forceinline__ int remap(int v, int m, int tlo, int thi) {
  int g = v + 3, r = m + 6, src = g;
  if (g < 3) {
    int j = 2 - g;
    src = (tlo == GP_BC_NEUMANN) ? 4 + j : r - 5 - j;
  } else if (g >= r - 3) {
    int j = g - (r - 3);
    src = (thi == GP_BC_NEUMANN) ? r - 5 - j : 4 + j;
  }
  return src - 3;
}

/* v / d for a divisor known in advance, r = RN(1/d): the correctly rounded
 * quotient in five multiply-adds (Markstein, "Computation of elementary functions
 * on the IBM RISC System/6000 processor", 1990, theorem on q' = RN(q + r * RN(v - d q)):
 * with r correctly rounded and q within one ulp of the quotient, q' is the
 * correctly rounded quotient).  The first pass brings v * r (off by up to 1.5 ulp)
 * within that; v outside [2^-900, 2^900) and not zero, where a product could
 * leave the normal range, takes the division, and so does every v when d is
 * outside [2^-60, 2^60) (span 0 instead of QUICK_SPAN, set on the host).  The interface tile of a 1.5-spaced grid spent half its time in
 * these divisions. */
/* out of line: inlined at every division it doubled the code of the tile */
static __device__ __noinline__ double slow_div(double v, double d) { return v / d; }
__device__ __forceinline__ double quick_div(double v, double d, double r, unsigned span) {
  const unsigned e = ((unsigned)__double2hiint(v) >> 20) & 0x7ffu;
  double q = v * r;
  if (e - 123u < span) {
    q = __fma_rn(__fma_rn(-q, d, v), r, q);
    q = __fma_rn(__fma_rn(-q, d, v), r, q);
  } else if (v != 0.0) {
    q = slow_div(v, d);
  }
  return q;
}
__device__ __forceinline__ float quick_div(float v, float d, float, unsigned) { return v / d; }
template <typename R>
__device__ __forceinline__ R divx(R v, const Consts<R> &D) {
  return D.mul_dx ? v * D.inv_dx : quick_div(v, D.dx, D.inv_dx, D.quick_span);
}
template <typename R>
__device__ __forceinline__ R divy(R v, const Consts<R> &D) {
  return D.mul_dy ? v * D.inv_dy : quick_div(v, D.dy, D.inv_dy, D.quick_span);
}
template <typename R>
__device__ __forceinline__ R div2y(R v, const Consts<R> &D) {
  return D.mul_dy ? v * D.inv_2dy : quick_div(v, R(2.0) * D.dy, D.inv_2dy, D.quick_span);
}

/* The same constants when every spacing is known to be a power of two (or
 * the field type is float): the divisions are multiplications by the exact
 * reciprocals and no division code is emitted.  Kernels view their Consts
 * through this type when the launch says so. */
template <typename R>
struct ConstsMul : Consts<R> {};
template <typename R>
__device__ __forceinline__ R divx(R v, const ConstsMul<R> &D) { return v * D.inv_dx; }
template <typename R>
__device__ __forceinline__ R divy(R v, const ConstsMul<R> &D) { return v * D.inv_dy; }
template <typename R>
__device__ __forceinline__ R div2y(R v, const ConstsMul<R> &D) { return v * D.inv_2dy; }

/* pair index of a<b among N phases */
template <int N>
__device__ __forceinline__ constexpr int pidx(int a, int b) {
  return a * N - a * (a + 1) / 2 + (b - a - 1);
}
template <int N>
struct NP { static constexpr int v = N * (N - 1) / 2 > 0 ? N * (N - 1) / 2 : 1; };

#define LI(i, j) ((i) * SW + (j))

/* Block-wide reduction helpers (deterministic order). */
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ double warp_min(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_down_sync(0xffffffffu, v, o));
  return v;
}

/* total order on doubles as signed 64-bit integers */
__device__ __forceinline__ long long ord(double v) {
  long long i = __double_as_longlong(v);
  return i < 0 ? i ^ 0x7fffffffffffffffLL : i;
}

/* Loads of what a step's kernels write: states, flags, lists, counters, temperature
 * rows.  The kernels of a step are launched while the one that writes these still
 * runs (pdl_begin, gp_fused.cuh), so they are not read-only for a kernel's lifetime:
 * no __ldg, no const __restrict__ pointer to them, and no load that the compiler
 * may move to before the wait (volatile, as the wait is). */
__device__ __forceinline__ double ld_step(const double *p) {
  double v;
  asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float ld_step(const float *p) {
  float v;
  asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ unsigned ld_step(const unsigned *p) {
  unsigned v;
  asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ int4 ld_step(const int4 *p) {
  int4 v;
  asm volatile("ld.global.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

struct StatBufs {
  long long *ext;      /* running extremes [simulations][2*(N+K)] (ordered ints, atomic max/min), or NULL */
  double *partials;    /* [tiles][2N+2K+1] sums when want_sums */
  int want_sums;
  const unsigned *round_step;  /* FP32 form: device step counter keying the rounding stream */
  int mbar_tries[2];   /* polls of such a box's barrier before the kernel gives up (MBAR_TRIES) */
  int bch_max, bch_div;  /* bulk chunks: at most bch_max (<= 16) entries, left / (bch_div * warps) */
  int mixed;           /* kf_step: odd CTAs take bulk tiles first, then interface tiles */
  const double *trows; /* non-isothermal simulations: per simulation the temperature of each ghosted column y
                          as the phase-field pass reads it, then as the concentration pass reads it */
  int sweep;           /* kf_bulk: a smoothing sweep's bulk tiles (no step is counted) */
  int diag;            /* every phase's off-diagonal D, c_mu and A are zero and no E is -0 */
  unsigned tma_extra[2];  /* bytes that the barrier of a bulk (MAP_MU) and of an interface tile's (MAP_ALL) box expects
                             beyond it: 0, or more to test the give-up paths */
  double *dphi_out;    /* NULL, or (a batch of one) the step's delta-phi of every interface tile and its ring in
                          the delta-phi layout (Grid dpitch/dplane); cells no interface tile covers are left as
                          they are (their delta-phi is +0.0) */
};

/* ---- FP32 storage rounding ------------------------------------------------
 * The FP32 form adds each step's increment in FP64 and rounds the sum to float
 * stochastically: up with probability (distance to the float below) / ulp.
 * Round-to-nearest would drop every increment below half an ulp (a slowly
 * diffusing far field stops moving and solute is lost); stochastic rounding
 * keeps every stored value unbiased, so the solute-mass error is a random walk
 * of size ulp*sqrt(steps/cells) instead of a systematic drift.  The random
 * bits are a counter-based hash of (step, cell, field): deterministic, and the
 * same for a simulation alone or inside a batch.  Values exactly
 * representable in float (pure phases 0/1, unchanged cells) are stored as is. */
__device__ __forceinline__ unsigned mix32(unsigned v) {
  /* a 32-bit avalanche hash (xor-shift / multiply rounds) */
  v ^= v >> 16;
  v *= 0x7feb352du;
  v ^= v >> 15;
  v *= 0x846ca68bu;
  v ^= v >> 16;
  return v;
}

__device__ __forceinline__ unsigned round_key(unsigned step, int x, int y) {
  return mix32(mix32(step * 0x9e3779b9u + 0x632be5abu) ^ ((unsigned)x * 0x85ebca6bu + (unsigned)y * 0xc2b2ae35u));
}

__device__ __forceinline__ float round_stochastic(double v, unsigned key, int field) {
  const float lo = __double2float_rz(v);              /* toward zero */
  const double rem = v - (double)lo;                   /* exact, same sign as v */
  if (rem == 0.0) return lo;
  const float hi = __uint_as_float(__float_as_uint(lo) + 1u);  /* next float away from zero */
  const double span = (double)hi - (double)lo;
  const double u = (double)(mix32(key + (unsigned)field * 0x27d4eb2fu) >> 8) * 0x1p-24;
  return fabs(rem) > u * fabs(span) ? hi : lo;
}

/* dmu = (dc/dmu)^-1 dc in FP64 by the simulation's inversion mode, and mu + dmu
 * into m64 (calculate_divergence_concentration.h:96-140) */
template <typename R, int K, typename CT>
__device__ __forceinline__ void solve_dmu(const CT &D, double (&dcdmu)[K][K], const double (&dc)[K], double (&m64)[K],
                                          double *dmu) {
#pragma unroll
  for (int k = 0; k < K; k++) dmu[k] = 0.0;
  if (D.inv_mode == GP_INV_BINARY) {
    double i00 = 1.0 / dcdmu[0][0];
    dmu[0] = dc[0] * i00;
    m64[0] += dmu[0];
  } else if (D.inv_mode == GP_INV_TERNARY && K == 2) {
    double det = dcdmu[0][0] * dcdmu[K - 1][K - 1] - dcdmu[0][K - 1] * dcdmu[K - 1][0];
    double iv[K][K];
    iv[0][0] = dcdmu[K - 1][K - 1] / det;
    iv[K - 1][K - 1] = dcdmu[0][0] / det;
    iv[0][K - 1] = -dcdmu[0][K - 1] / det;
    iv[K - 1][0] = -dcdmu[K - 1][0] / det;
#pragma unroll
    for (int k = 0; k < K; k++) {
      dmu[k] = 0.0;
#pragma unroll
      for (int l = 0; l < K; l++) dmu[k] += iv[k][l] * dc[l];
    }
#pragma unroll
    for (int k = 0; k < K; k++) m64[k] = dmu[k] + m64[k];
  } else if (D.inv_mode == GP_INV_DILUTE) {
#pragma unroll
    for (int k = 0; k < K; k++) {
      double ikk = 1.0 / dcdmu[k][k];
      dmu[k] = dc[k] * ikk;
      m64[k] += dmu[k];
    }
  } else {
    double iv[K][K];
    matinv_div<double, K>(dcdmu, iv);
#pragma unroll
    for (int k = 0; k < K; k++) {
      double s = 0;
#pragma unroll
      for (int l = 0; l < K; l++) s = s + iv[k][l] * dc[l];
      dmu[k] = s;
    }
#pragma unroll
    for (int k = 0; k < K; k++) m64[k] = dmu[k] + m64[k];
  }
}

/* ------------------------------------------------------------------ */
/* batched simulations                                                 */
/* ------------------------------------------------------------------ */

/* One simulation of a batch: its geometry, where its planes start in the
 * pooled buffers, and its tiles in the batch's tile numbering. */
struct SimDesc {
  Grid g;
  long long off_state;   /* N phi planes then K mu planes */
  int tiles_x, tile0;    /* tiles per row, first tile */
  int off_T;             /* non-isothermal: the step's temperature rows (two of MESH_Y+6) in StatBufs::trows */
};

}  // namespace gpd
