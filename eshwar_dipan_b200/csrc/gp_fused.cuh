/*
 * gp_fused.cuh -- the time step as kernels over classified tiles.
 *
 * Every TX x TY tile of every simulation carries a phase flag per state
 * buffer: p >= 0 when each of its cells holds exactly the one-hot phi of phase
 * p (bits of 1.0 and +0.0), -1 otherwise, -2 when not known.  A tile whose own
 * flag and the flags of every tile its two-cell phi halo reaches (through the
 * boundary copy tables) are the same p >= 0 is a bulk tile: no phase is
 * active anywhere on its delta-phi ring (every Laplacian is 0.0), so delta-phi
 * is +0.0 there, no anti-trapping current flows, every cell takes the bulk
 * branch of the mu update with the pure-phase D, and phi stays as it is
 * (calculate_divergence_phasefield.h:19-22, calculate_fluxes_concentration.h:64,
 * calculate_divergence_concentration.h:43-57).
 *
 *  kf_classify one thread per tile: the bulk test; bulk and interface lists.
 *  kf_bulk     persistent warps over contiguous ranges of the bulk list, the
 *              next tile's mu in flight (one TMA box) while one is stepped.  Bulk
 *              tiles read and write mu only (phi is rewritten only when the
 *              output buffer does not already hold the same one-hot tile).
 *  kf_general  persistent CTAs over the interface list (gp_iface.cuh): delta-phi
 *              on a tile plus its one-cell ring in shared memory (the ring is
 *              recomputed by each neighbour instead of going through HBM), then
 *              the mu update and the phi commit, and the tile's new flags.
 *
 * The arithmetic of each cell is the reference's, in its order (FP64 results
 * are bit-identical to the reference step); the FP32 form differs only where
 * gp_tiles.cuh says.
 */
#pragma once
#include <climits>
#include <type_traits>

#include "gp_iface.cuh"
#include "gp_iface32.cuh"
#include "gp_tiles.cuh"

namespace gpd {

constexpr signed char FLAG_MIXED = -1, FLAG_UNKNOWN = -2;

/* A pair of floats in one 64-bit register pair, for sm_100's packed FP32
 * arithmetic (add/sub/mul/fma .rn.f32x2: two IEEE single-precision results,
 * round to nearest, per instruction). */
typedef unsigned long long f2;
__device__ __forceinline__ f2 f2pack(float lo, float hi) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float f2lo(f2 v) {
  float lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
  return lo;
}
__device__ __forceinline__ float f2hi(f2 v) {
  float lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
  return hi;
}
__device__ __forceinline__ f2 f2add(f2 a, f2 b) {
  f2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2 f2sub(f2 a, f2 b) {
  f2 d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2 f2mul(f2 a, f2 b) {
  f2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2 f2fma(f2 a, f2 b, f2 c) {
  f2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
/* three-operand max/min (a NaN operand is ignored, as by fmaxf) */
__device__ __forceinline__ float fmax3f(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float fmin3f(float a, float b, float c) {
  float d;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
/* spacing of the floats at |v| (2^(e-23) for a normal v of exponent e; the
 * subnormal spacing below) */
__device__ __forceinline__ float ulpf(float v) {
  const unsigned e = max(__float_as_uint(v) & 0x7f800000u, 24u << 23);
  return __uint_as_float(e - (23u << 23));
}

/* Phase flags of one tile in one state buffer: for the whole tile and for its
 * four two-cell-deep edge bands (top = first two rows, bot = last two rows,
 * left/right = first/last two columns, over the tile's cells inside the
 * domain): the phase p whose exact one-hot phi every cell of the region holds,
 * FLAG_MIXED, or FLAG_UNKNOWN.  8 bytes, read as one word.  The bottom and
 * right bands are read only where a tile follows (the tile is then full). */
struct __align__(8) TileFlags {
  signed char whole, top, bot, left, right, pad0, pad1, pad2;
};

/* one-hot test on exact bits: phase index, or -1 */
template <typename R, int N>
__device__ __forceinline__ int one_hot(const R *ph) {
  int p = -1, ones = 0, zeros = 0;
#pragma unroll
  for (int a = 0; a < N; a++) {
    if (sizeof(R) == 8) {
      const long long b = __double_as_longlong((double)ph[a]);
      if (b == 0x3ff0000000000000LL) { p = a; ones++; }
      else if (b == 0) zeros++;
    } else {
      const unsigned b = __float_as_uint((float)ph[a]);
      if (b == 0x3f800000u) { p = a; ones++; }
      else if (b == 0u) zeros++;
    }
  }
  return (ones == 1 && zeros == N - 1) ? p : -1;
}

/* Flag bits of one tile row (a warp, a lane per column) from the one-hot phase
 * (or -1) of each lane's cell: bit p: every valid cell holds phase p; bit 8+p:
 * those of the first two columns; bit 16+p: those of the last two.  Call with the
 * whole warp. */
template <int N>
__device__ __forceinline__ unsigned row_flag_bits(bool valid, int oh) {
  const unsigned v = __ballot_sync(0xffffffffu, valid);
  unsigned r = 0;
#pragma unroll
  for (int p = 0; p < N; p++) {
    const unsigned miss = v & ~__ballot_sync(0xffffffffu, oh == p);
    r |= (miss ? 0u : 1u << p) | ((miss & 0x3u) ? 0u : 1u << (8 + p)) |
         ((miss & 0xc0000000u) ? 0u : 1u << (16 + p));
  }
  return r;
}
/* a tile's flags from its rows' bits; a row outside the domain holds every bit */
__device__ __forceinline__ TileFlags flags_of_rows(const unsigned *w) {
  unsigned all = w[0];
#pragma unroll
  for (int r = 1; r < TX; r++) all &= w[r];
  auto phase = [](unsigned bits) { return bits ? (signed char)(__ffs(bits) - 1) : FLAG_MIXED; };
  TileFlags t;
  t.whole = phase(all & 0xffu);
  t.top = phase(w[0] & w[1] & 0xffu);
  t.bot = phase(w[TX - 2] & w[TX - 1] & 0xffu);
  t.left = phase((all >> 8) & 0xffu);
  t.right = phase((all >> 16) & 0xffu);
  t.pad0 = t.pad1 = t.pad2 = 0;
  return t;
}

__device__ __forceinline__ TileFlags ld_step(const TileFlags *p) {
  union {
    unsigned long long w;
    TileFlags t;
  } v;
  asm volatile("ld.global.u64 %0, [%1];" : "=l"(v.w) : "l"(p));
  return v.t;
}

__device__ __forceinline__ TileFlags uniform_flags(int p) {
  TileFlags t;
  t.whole = t.top = t.bot = t.left = t.right = (signed char)p;
  t.pad0 = t.pad1 = t.pad2 = 0;
  return t;
}

/* what the classification needs of a simulation (phi's boundary types); tiles_x 0: a
 * batch of several, read from their descriptors */
struct ClassifySim {
  int mx, my, tiles_x, bc_x[2], bc_y[2], tgrad;
};

/* Bulk test of tile (tile rows by, columns bx) of a simulation, by one
 * thread: every cell of the tile and of its two-cell phi halo holds the exact
 * one-hot phi of one phase.  Returns the phase or -1.  When the halo stays
 * inside the domain it is covered by the facing edge bands of the eight
 * neighbour tiles (a corner by either band that contains it); otherwise by the
 * whole-tile flags of the tiles that hold the halo cells after the boundary
 * remap. */
__device__ __forceinline__ int bulk_phase(const ClassifySim &g, const TileFlags *flags, int tile0, int by,
                                          int bx) {
  const int tiles_x = g.tiles_x;
  const int x0 = by * TX, y0 = bx * TY;
  const int xl = min(x0 + TX, g.mx) - 1, yl = min(y0 + TY, g.my) - 1;
  if (x0 >= 2 && xl + 2 < g.mx && y0 >= 2 && yl + 2 < g.my) {
    const TileFlags *f = flags + tile0 + by * tiles_x + bx;
    const TileFlags ul = ld_step(f - tiles_x - 1), u = ld_step(f - tiles_x), ur = ld_step(f - tiles_x + 1);
    const TileFlags l = ld_step(f - 1), c = ld_step(f), r = ld_step(f + 1);
    const TileFlags dl = ld_step(f + tiles_x - 1), d = ld_step(f + tiles_x), dr = ld_step(f + tiles_x + 1);
    const int p = c.whole;
    const bool ok = p >= 0 && u.bot == p && d.top == p && l.right == p && r.left == p &&
                    (ul.bot == p || ul.right == p) && (ur.bot == p || ur.left == p) &&
                    (dl.top == p || dl.right == p) && (dr.top == p || dr.left == p);
    return ok ? p : -1;
  }
  /* the tiles of rows x0-2, x0-1, xl+1, xl+2 and columns y0-2, y0-1, yl+1, yl+2 */
  int rows[5], cols[5];
  {
    const int xs[4] = {x0 - 2, x0 - 1, xl + 1, xl + 2};
    const int ys[4] = {y0 - 2, y0 - 1, yl + 1, yl + 2};
    rows[0] = by;
    cols[0] = bx;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      int x = xs[q], y = ys[q];
      if (x < 0 || x >= g.mx) x = remap(x, g.mx, g.bc_x[0], g.bc_x[1]);
      if (y < 0 || y >= g.my) y = remap(y, g.my, g.bc_y[0], g.bc_y[1]);
      rows[q + 1] = x / TX;
      cols[q + 1] = y / TY;
    }
  }
  int w[25];   /* all loads first: one after the other they would be a chain */
#pragma unroll
  for (int q = 0; q < 25; q++) w[q] = ld_step(flags + tile0 + rows[q / 5] * tiles_x + cols[q % 5]).whole;
  const int p = w[0];   /* the tile itself */
  bool ok = p >= 0;
#pragma unroll
  for (int q = 1; q < 25; q++) ok = ok & (w[q] == p);
  return ok ? p : -1;
}


/* ------------------------------------------------------------------ */
/* kernels                                                             */
/* ------------------------------------------------------------------ */

/* Work-list counters of a batch: [0] interface tiles listed by kf_classify,
 * [1] interface entries taken beyond the CTAs' first, [2] CTAs of the step's kernels
 * finished, [3] step number (keys the FP32 rounding stream), [4] bulk tiles
 * listed, [5] error flag (a TMA box did not arrive; the host reads and clears it),
 * [6] bulk entries taken.  A step is kf_classify, then kf_step or kf_bulk and
 * kf_general; the last CTA after kf_classify resets [0..2], [4] and [6] and
 * advances [3]. */
enum { CTR_LIST = 0, CTR_HEAD = 1, CTR_DONE = 2, CTR_STEP = 3, CTR_BULK = 4, CTR_ERR = 5, CTR_BHEAD = 6,
       CTR_COUNT = 8 };

/* Programmatic dependent launch: the kernels of a step are launched while their
 * predecessor still runs (every one of its CTAs has started) and wait here, before
 * they read anything it writes (with ld_step only), until it has completed.  A launch gap of a graph
 * is about 1 us; a step has two.  Large single grids lose by it and launch in order
 * (GP_PLAIN_TILES, gp_device.cu, has both sides' times); the wait is then no wait. */
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_begin() {
  pdl_launch();
  pdl_wait();
}

/* End of one CTA of the step's bulk or interface kernel (they may run
 * concurrently): the last of the step's ndone CTAs empties the lists and
 * advances the step counter by `steps` (0: a smoothing sweep).  Call with all
 * threads. */
__device__ __forceinline__ void step_finish(int *ctr, int ndone, int steps) {
  __shared__ int s_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(ctr + CTR_DONE, 1) == ndone - 1;
  }
  __syncthreads();
  if (s_last && threadIdx.x == 0) {
    ctr[CTR_LIST] = 0;
    ctr[CTR_HEAD] = 0;
    ctr[CTR_DONE] = 0;
    ctr[CTR_BULK] = 0;
    ctr[CTR_BHEAD] = 0;
    ctr[CTR_STEP] = (int)((unsigned)ctr[CTR_STEP] + (unsigned)steps);
    __threadfence();
  }
}

/* One thread per tile: the bulk test, then the tile goes on the bulk list
 * or the interface list; one atomic per warp and list.  A bulk entry holds
 * everything kf_bulk needs to start the tile: {t | phase << 28, simulation |
 * flag of the output buffer << 24, tile row << 16 | tile column, 0}; an interface
 * entry {t, simulation, tile row << 16 | tile column, 1 when the tile is full and
 * its two-cell halo lies inside the domain (staged by one TMA box)}.  Small CTAs
 * (NTC threads) spread the flag reads over every SM. */
constexpr int NTC = 64;
template <typename R>
__global__ void __launch_bounds__(NTC) kf_classify(const ClassifySim solo, const SimDesc *__restrict__ sims,
                                                  const Consts<R> *__restrict__ consts, const int *__restrict__ tsim,
                                                  int ntiles, const TileFlags *flag_in,
                                                  const TileFlags *flag_outbuf,
                                                  int4 *__restrict__ glist, int4 *__restrict__ blist,
                                                  int *__restrict__ ctr) {
  const int t = blockIdx.x * NTC + threadIdx.x, lane = threadIdx.x & 31;
  int p = -1, s = 0, by = 0, bx = 0, inside = 0;
  if (solo.tiles_x) {
    /* a batch of one: its layout comes with the launch */
    by = t / solo.tiles_x;
    bx = t - by * solo.tiles_x;
  }
  pdl_begin();
  if (t < ntiles) {
    ClassifySim cs = solo;
    int tile0 = 0;
    if (!solo.tiles_x) {
      s = __ldg(tsim + t);
      const SimDesc &sd = sims[s];
      const Consts<R> &D = consts[s];
      cs = {sd.g.mx, sd.g.my, sd.tiles_x, {D.bc_x[0][0], D.bc_x[0][1]}, {D.bc_y[0][0], D.bc_y[0][1]}, D.tgrad};
      tile0 = sd.tile0;
      by = (t - tile0) / cs.tiles_x;
      bx = t - tile0 - by * cs.tiles_x;
    }
    inside = by > 0 && by * TX + TX + 2 <= cs.mx && bx > 0 && bx * TY + TY + 2 <= cs.my;
    /* a non-isothermal simulation steps every tile as an interface tile
     * (whose pure-phase cells take the bulk update at their temperature) */
    if (!cs.tgrad) p = bulk_phase(cs, flag_in, tile0, by, bx);
  }
  const unsigned mb = __ballot_sync(0xffffffffu, t < ntiles && p >= 0);
  const unsigned mg = __ballot_sync(0xffffffffu, t < ntiles && p < 0);
  int bb = 0, bg = 0;
  if (lane == 0) {
    if (mb) bb = atomicAdd(ctr + CTR_BULK, __popc(mb));
    if (mg) bg = atomicAdd(ctr + CTR_LIST, __popc(mg));
  }
  bb = __shfl_sync(0xffffffffu, bb, 0);
  bg = __shfl_sync(0xffffffffu, bg, 0);
  const unsigned below = (1u << lane) - 1u;
  if (t < ntiles) {
    if (p >= 0)
      blist[bb + __popc(mb & below)] =
          make_int4(t | (p << 28), s | (((int)ld_step(flag_outbuf + t).whole & 0xff) << 24), (by << 16) | bx, 0);
    else
      glist[bg + __popc(mg & below)] = make_int4(t, s, (by << 16) | bx, inside);
  }
}

/* ---- TMA and mbarrier primitives (one CTA, no cluster, no multicast) ---- */
__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
}
/* make barrier initialisation and earlier generic shared-memory writes
 * visible to the async (TMA) proxy */
__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
/* tiled 3-D tensor copy global -> this CTA's shared memory, completion
 * counted in bytes on bar; c0 is the innermost coordinate */
__device__ __forceinline__ void tma_load_3d(unsigned dst, const void *tmap, int c0, int c1, int c2, unsigned bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
      "[%5];\n" ::"r"(dst),
      "l"(tmap), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
      : "memory");
}
__device__ __forceinline__ bool mbar_test(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
/* wait for phase `parity` of bar to complete, at most `tries` polls (each
 * poll may suspend the thread for a short while); false when it did not */
constexpr int MBAR_TRIES = 1 << 20;
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity, int tries) {
  for (int it = 0; it < tries; it++)
    if (mbar_test(bar, parity)) return true;
  return false;
}

/* eight bytes of global memory into shared memory, asynchronously (n = 0: zeros) */
__device__ __forceinline__ void cp_async8(void *dst, const void *src, unsigned n) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

/* x/dx and y/dy of the bulk kernel: a multiplication by the reciprocal when
 * the spacing is a power of two (MUL, chosen at launch), else the division */
template <bool MUL, typename R>
__device__ __forceinline__ R bdiv(R v, R inv, R d, unsigned span) {
  if constexpr (MUL) return v * inv;
  else return quick_div(v, d, inv, span);
}

/* Tensor maps (CUtensorMap, 128 bytes), two per simulation and state buffer:
 * MAP_MU of the K mu planes, dimensions {pitch, mx, K}, box {BulkGeom::BW, SH, K}
 * (bulk tiles); MAP_ALL of the N + K planes, box {ItemGeom::BW, FR, N + K}
 * (interface items). */
enum { MAP_MU = 0, MAP_ALL = 1, MAP_KINDS = 2 };
struct alignas(64) TensorMapSlot {
  unsigned long long w[16];
};

/* The maps of a batch of one (nsims 1), for the buffer a launch reads: they come as
 * a kernel parameter, where the launch itself makes them current.  A batch of
 * several reads them from global memory. */
struct BoxMaps {
  TensorMapSlot m[MAP_KINDS];
  int nsims;
  int ahead;   /* a batch of several: every block fences all maps before its wait */
};

/* The copy unit keeps descriptors it has read; one in global memory may be an older
 * one's from the same address until a block has fenced it.  The host writes the maps
 * once, before any step.  So every block may fence all of them ahead of its wait,
 * while the kernel before finishes, which costs by the simulations; or a thread fences
 * a map when it moves to its simulation, which costs by the tiles.  Step times, ahead /
 * at each move: 24 simulations of 128^2 to 1024^2 82 / 89 us, 64 of 256^2 50 / 54 us,
 * 256 of 128^2 to 1024^2 262 / 265 us, 256 of 256^2 148 / 148 us, 256 of 128^2 110 / 103 us,
 * 1024 of 64^2 443 / 380 us (FP32; FP64 alike): ahead from as many tiles as the
 * simulations squared (box_fence_ahead). */
__host__ __device__ __forceinline__ bool box_fence_ahead(long long nsims, long long ntiles) {
  return nsims > 1 && ntiles >= nsims * nsims;
}
__device__ __forceinline__ void box_fence(const TensorMapSlot *m) {
  asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(m) : "memory");
}
/* Start of a kernel that issues boxes of the kinds in KINDS (bit k: kind k).  SOLO: a
 * batch of one. */
template <unsigned KINDS, bool SOLO>
__device__ __forceinline__ void box_begin(const BoxMaps &maps, const TensorMapSlot *tmaps, int buf) {
  pdl_launch();
  if (!SOLO && maps.ahead) {
    for (int s = threadIdx.x; s < maps.nsims; s += NTI) {
#pragma unroll
      for (int k = 0; k < MAP_KINDS; k++)
        if ((KINDS >> k) & 1u) box_fence(tmaps + (2 * s + buf) * MAP_KINDS + k);
    }
    __syncthreads();
  }
  pdl_wait();
}
/* the map of a box of simulation s, after box_begin, to be used by the calling thread
 * (ready: the map that it fenced last) */
__device__ __forceinline__ const TensorMapSlot *box_map(const BoxMaps &maps, const TensorMapSlot *tmaps, int s, int buf,
                                                        int kind, const TensorMapSlot *&ready) {
  if (maps.nsims == 1) return &maps.m[kind];
  const TensorMapSlot *const m = tmaps + (2 * s + buf) * MAP_KINDS + kind;
  if (!maps.ahead && m != ready) {
    box_fence(m);
    ready = m;
  }
  return m;
}

/* Shared memory of one warp of kf_bulk: NST stages of mu with a one-cell halo,
 * each filled by one TMA box.  A box starts CO columns left of the halo
 * column so that its first column is 16-byte aligned (y0 - 1 - CO is a
 * multiple of 16 bytes / sizeof(R)); stage column c holds y = y0 - 1 - CO + c. */
template <typename R, int K>
struct BulkGeom {
  static constexpr int CO = sizeof(R) == 8 ? 1 : 3;
  static constexpr int BW = SW + 2 * CO;   /* 36 doubles or 40 floats: a multiple of 16 bytes */
  /* boxes in flight per warp: 4 of FP32 or 2 of FP64 (the same bytes) */
  static constexpr int NST = sizeof(R) == 4 ? 4 : 2;
  static constexpr unsigned BOX_BYTES = (unsigned)(K * SH * BW * sizeof(R));
};
template <typename R, int K>
struct alignas(128) BulkStage {
  R M[K][SH][BulkGeom<R, K>::BW];
};
/* list entry of a tile in flight: tile | phase << 28, simulation, first
 * cell, the flag of its output buffer */
struct BulkEntry {
  int item, s, x0, y0, have;
};
template <typename R, int K>
struct alignas(128) BulkWarpSmem {
  BulkStage<R, K> st[BulkGeom<R, K>::NST];
  unsigned long long bar[BulkGeom<R, K>::NST];
  BulkEntry meta[BulkGeom<R, K>::NST];
};
/* dynamic shared memory of kf_bulk */
template <typename R, int K>
constexpr size_t bulk_smem_bytes() {
  return (NTI / 32) * sizeof(BulkWarpSmem<R, K>);
}
/* The step kernels' dynamic shared memory (TMA boxes want 128-byte alignment).
 * Named in every function that uses it, so that its accesses are shared-memory
 * loads and stores: through a pointer argument, or a base rounded up as an
 * integer, they were generic ones with 64-bit address arithmetic. */
extern __shared__ __align__(128) unsigned char step_smem_base[];

/* The FP64 bulk update of one cell (stage row i, column j) of phase p with
 * every term of the K x K matrices: the expressions of a non-DIAG kernel in
 * their order (calculate_divergence_concentration.h:43-57 through
 * functionF_01.h:19-37).  A DIAG kernel calls it, after a tile's rows, for
 * the rare cells whose result was not finite. */
template <int K, bool MUL>
__device__ __forceinline__ void bulk_cell_full_f64(const double *__restrict__ st, int i, int j,
                                                const Consts<double> *__restrict__ Dp, int p, const double *m,
                                                double *nm, double *dmu) {
  constexpr int BW = BulkGeom<double, K>::BW;
  const Consts<double> &D = *Dp;
  const double idx = D.inv_dx, idy = D.inv_dy, ddx = D.dx, ddy = D.dy, dt = D.dt;
  const unsigned qs = D.quick_span;
  const double cst = D.obstacle ? D.jat_obst : D.jat_well;
  double divjat = bdiv<MUL>((0.0 - 0.0) * cst, idx, ddx, qs);
  divjat += bdiv<MUL>((0.0 - 0.0) * cst, idy, ddy, qs);
#define BM(l, r, c) st[((l) * SH + (r)) * BW + (c)]
  double cn[K];
#pragma unroll
  for (int k = 0; k < K; k++) {
    double divflux = 0.0;
#pragma unroll
    for (int l = 0; l < K; l++) {
      const double Dv = D.Dbulk[p][k][l];
      const double dm = (Dv + Dv) * 0.5, c = BM(l, i, j);
      const double fx = dm * bdiv<MUL>(BM(l, i + 1, j) - c, idx, ddx, qs);
      const double bx_ = dm * bdiv<MUL>(c - BM(l, i - 1, j), idx, ddx, qs);
      const double fy = dm * bdiv<MUL>(BM(l, i, j + 1) - c, idy, ddy, qs);
      const double by_ = dm * bdiv<MUL>(c - BM(l, i, j - 1), idy, ddy, qs);
      divflux += bdiv<MUL>(fx - bx_, idx, ddx, qs);
      divflux += bdiv<MUL>(fy - by_, idy, ddy, qs);
    }
    double cm = 0.0;   /* c_mu (functionF_01.h:30-37) */
#pragma unroll
    for (int l = 0; l < K; l++) cm += D.cmu[p][k][l] * (m[l] - D.E[p][l]);
    cn[k] = cm + dt * (divflux) - divjat;
  }
#undef BM
#pragma unroll
  for (int k = 0; k < K; k++) {
    double sm = D.twoA[p][k] * cn[k] + D.E[p][k];   /* Mu (functionF_01.h:19-29) */
#pragma unroll
    for (int l = 0; l < K; l++)
      if (k != l) sm += D.A[p][k][l] * cn[l];
    nm[k] = sm;
    dmu[k] = sm - m[k];
  }
}

/* Bulk tiles, one warp per tile.  Warps take contiguous ranges of the bulk
 * list.  Lane 0 issues one TMA box per tile (the K mu planes of the tile with
 * a one-cell halo, rows x0-1..x0+TX) into the warp's next stage while the warp
 * steps the current one; an mbarrier per stage counts the bytes in.  Halo
 * cells outside the domain (tiles on the boundary) are then overwritten with
 * the cells the boundary copy tables name.  Lane j steps column y0+j row by
 * row.  No block-wide barrier anywhere.  The running mu extremes of the cells
 * a warp steps stay in registers and are merged into the simulation's slots
 * (atomic max/min) when the warp moves to another simulation or finishes;
 * bulk tiles cannot move the phi extremes (their phi is 0 or 1, inside the
 * initial [0, 1]).  A stage whose bytes do not arrive within the poll limit
 * sets ctr[CTR_ERR]; the warp then stops taking tiles.  A call of its own: inlined
 * beside the interface code it made both spill. */
template <typename R, int N, int K, bool SUMS, bool MUL, bool DIAG>
__device__ __noinline__ void bulk_tiles(const SimDesc *__restrict__ sims, const Consts<R> *__restrict__ consts,
                                           const int4 *blist, const BoxMaps &maps,
                                           const TensorMapSlot *__restrict__ tmaps, int buf,
                                           const R *state, R *__restrict__ next,
                                           TileFlags *__restrict__ flag_out, int *__restrict__ ctr,
                                           const StatBufs st) {
  using G = BulkGeom<R, K>;
  constexpr int NS = 2 * N + 2 * K + 1, NST = G::NST, CO = G::CO;
  BulkWarpSmem<R, K> &ws = reinterpret_cast<BulkWarpSmem<R, K> *>(step_smem_base)[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const int nbulk = *(const volatile int *)(ctr + CTR_BULK);

  if (lane == 0) {
#pragma unroll
    for (int q = 0; q < NST; q++) mbar_init(smem_addr(&ws.bar[q]), 1);
    fence_barrier_init();
    fence_proxy_async_smem();
  }
  __syncwarp();

  /* Running mu extremes of the cells a lane stepped.  FP64: they start at the
   * simulation's extremes as they were when the warp moved to it (kept finite, so
   * that an infinity exceeds them), and a row takes the slow way only where a value
   * does: two comparisons a value where fmax and fmin took about eight instructions
   * each, a quarter of the kernel's.  FP32 (three-operand max and min): from
   * infinities. */
  constexpr bool F64 = sizeof(R) == 8;
  R emax[K], emin[K];
#pragma unroll
  for (int k = 0; k < K; k++) { emax[k] = -INFINITY; emin[k] = INFINITY; }
  bool beaten = !F64;
  int cur_sim = -1;
  auto ext_slot = [&](int s) { return st.ext + (long long)s * (2 * (N + K)) + 2 * N; };   /* max mu[K], min mu[K] */
  auto from_ord = [](long long o) { return __longlong_as_double(o < 0 ? o ^ 0x7fffffffffffffffLL : o); };
  auto flush = [&](int s) {
    if (__any_sync(0xffffffffu, beaten)) {
#pragma unroll
      for (int k = 0; k < K; k++) {
        const double a = warp_max(emax[k]), c = warp_min(emin[k]);
        if (lane == 0 && st.ext) {
          long long *slot = ext_slot(s);
          /* an extreme that is already there takes no atomic */
          if (a > from_ord(*(volatile long long *)(slot + k))) atomicMax(slot + k, ord(a));
          if (c < from_ord(*(volatile long long *)(slot + K + k))) atomicMin(slot + K + k, ord(c));
        }
      }
    }
#pragma unroll
    for (int k = 0; k < K; k++) { emax[k] = -INFINITY; emin[k] = INFINITY; }
    beaten = !F64;
  };
  auto load_ext = [&](int s) {
    if constexpr (F64) {
#pragma unroll
      for (int k = 0; k < K; k++) {
        emax[k] = 1.7976931348623157e308;    /* without a record nothing finite exceeds them */
        emin[k] = -1.7976931348623157e308;
        if (st.ext) {
          emax[k] = fmin(emax[k], from_ord(*(volatile long long *)(ext_slot(s) + k)));
          emin[k] = fmax(emin[k], from_ord(*(volatile long long *)(ext_slot(s) + K + k)));
        }
      }
    }
  };

  /* Work comes in chunks of list entries taken from the bulk head counter
   * (one atomic per warp and chunk), so warps that run faster take more; the
   * chunk size shrinks as the list drains (a few chunks per warp in all; the
   * batch's launch shape sets the largest chunk and the divisor).
   * Two chunks are held: A (being issued) and B (next).  Lane h*16+r holds
   * entry r of the chunk in half h; B's entries are loaded when it is taken,
   * one 16-byte load per lane, and used one tile later. */
  constexpr int BCH = 16;
  const int nwarps = gridDim.x * (NTI / 32);
  int q_item = 0, q_s = 0, q_xy = 0;   /* q_s: simulation | output flag << 24; q_xy: tile row << 16 | column */
  auto grab = [&](int half, int &start, int &n) {
    int v = 0, c = 0;
    if (lane == 0) {
      const int left = nbulk - *(volatile int *)(ctr + CTR_BHEAD);
      c = max(2, min(min(BCH, st.bch_max), left / (st.bch_div * nwarps)));
      v = atomicAdd(ctr + CTR_BHEAD, c);
    }
    start = __shfl_sync(0xffffffffu, v, 0);
    c = __shfl_sync(0xffffffffu, c, 0);
    n = max(0, min(c, nbulk - start));
    const int r = lane - 16 * half;
    if (r >= 0 && r < n) {
      const int4 e = ld_step(blist + start + r);
      q_item = e.x;
      q_s = e.y;
      q_xy = e.z;
    }
  };
  int ha = 0, na = 0, pa = 0;   /* chunk A: half, entries, next to issue */
  int cb = 0, nb = 0;           /* chunk B (half ha ^ 1) */
  {
    int ca = 0;
    grab(0, ca, na);
  }
  if (na > 0) grab(1, cb, nb);
  /* the next entry in issue order; false when the list is used up */
  auto next_entry = [&](BulkEntry &en) {
    if (pa == na) {
      if (nb == 0) return false;
      ha ^= 1;
      na = nb;
      pa = 0;
      grab(ha ^ 1, cb, nb);
    }
    const int r = 16 * ha + pa;
    en.item = __shfl_sync(0xffffffffu, q_item, r);
    const int sh = __shfl_sync(0xffffffffu, q_s, r), xy = __shfl_sync(0xffffffffu, q_xy, r);
    en.s = sh & 0xffffff;
    en.have = (signed char)(sh >> 24);
    en.x0 = (xy >> 16) * TX;
    en.y0 = (xy & 0xffff) * TY;
    pa++;
    return true;
  };
  const TensorMapSlot *ready = nullptr;
  /* lane 0: start the TMA box of a tile into stage b and note its entry */
  auto issue = [&](const BulkEntry &en, int b) {
    if (lane == 0) {
      ws.meta[b] = en;
      const unsigned bar = smem_addr(&ws.bar[b]);
      mbar_expect_tx(bar, G::BOX_BYTES + st.tma_extra[MAP_MU]);
      tma_load_3d(smem_addr(&ws.st[b]), box_map(maps, tmaps, en.s, buf, MAP_MU, ready), en.y0 - 1 - CO, en.x0 - 1, 0, bar);
    }
  };

  /* the current simulation's layout and the current (simulation, phase)'s
   * constants stay in registers while consecutive tiles share them */
  Grid g = {};
  long long off_state = 0;
  int cur_key = -1;
  unsigned qs = 0;
  R idx = R(0), idy = R(0), ddx = R(1), ddy = R(1), dt = R(0), divjat = R(0);
  /* the K x K constants of a phase: diffusive flux factor, c_mu, A and
   * dmu/dc */
  struct MatC {
    R dm[K][K], cmu[K][K], A[K][K], muc[K][K];
  };
  auto load_mat = [&](MatC &c, const Consts<R> &D, int p) {
#pragma unroll
    for (int k = 0; k < K; k++)
#pragma unroll
      for (int l = 0; l < K; l++) {
        const R Dv = D.Dbulk[p][k][l];
        c.dm[k][l] = (Dv + Dv) * R(0.5);
        c.cmu[k][l] = D.cmu[p][k][l];
        c.A[k][l] = D.A[p][k][l];
        c.muc[k][l] = (R)D.muc64[p][k][l];
      }
  };
  R E[K], twoA[K];
  MatC mc;
  /* FP32: flux-divergence coefficients of the bulk update (x and y) */
  f2 CX2[K][K], CY2[K][K];
  /* FP32: the step's part of the rounding key */
  const unsigned skey = sizeof(R) == 4 ? mix32(ld_step(st.round_step) * 0x9e3779b9u + 0x632be5abu) : 0u;

  /* the qi-th box a warp issues goes to stage qi % NST and completes phase
   * (qi / NST) & 1 of that stage's barrier; NST-1 boxes are in flight while a
   * tile is stepped */
  int qi = 0, ci = 0;
  for (int q = 0; q < NST - 1; q++) {
    BulkEntry en;
    if (!next_entry(en)) break;
    issue(en, qi % NST);
    qi++;
  }
  __syncwarp();
  while (ci < qi) {
    {
      BulkEntry en;
      if (next_entry(en)) {   /* into the stage of tile ci-1, stepped already */
        issue(en, qi % NST);
        qi++;
      }
    }
    const int b = ci % NST;
    if (!mbar_wait(smem_addr(&ws.bar[b]), (ci / NST) & 1, st.mbar_tries[MAP_MU])) {
      /* bytes missing: record it, wait (bounded) for the other boxes in
       * flight, step nothing more */
      if (lane == 0) atomicExch(ctr + CTR_ERR, 1);
      for (int q = ci + 1; q < qi; q++) mbar_wait(smem_addr(&ws.bar[q % NST]), (q / NST) & 1, st.mbar_tries[MAP_MU]);
      break;
    }
    ci++;
    /* ---- step bulk tile t (phase p) from stage b */
    const BulkEntry cur = ws.meta[b];
    const int t = cur.item & 0x0fffffff, p = cur.item >> 28, s = cur.s;
    const int x0 = cur.x0, y0 = cur.y0, have = cur.have;
    const Consts<R> &D = consts[s];
    if (s != cur_sim) {
      if (cur_sim >= 0) flush(cur_sim);
      cur_sim = s;
      g = sims[s].g;
      off_state = sims[s].off_state;
      load_ext(s);
    }
    if (cur_key != s * 16 + p) {
      cur_key = s * 16 + p;
      idx = D.inv_dx; idy = D.inv_dy; ddx = D.dx; ddy = D.dy; dt = D.dt; qs = D.quick_span;
      const R cst = D.obstacle ? D.jat_obst : D.jat_well;
      /* the anti-trapping divergence of a bulk cell: no phi gradient, the
       * same value for every cell */
      divjat = bdiv<MUL>((R(0.0) - R(0.0)) * cst, idx, ddx, qs);
      divjat += bdiv<MUL>((R(0.0) - R(0.0)) * cst, idy, ddy, qs);
#pragma unroll
      for (int k = 0; k < K; k++) {
        E[k] = D.E[p][k];
        twoA[k] = D.twoA[p][k];
      }
      /* a DIAG kernel keeps only the diagonals live */
      load_mat(mc, D, p);
      if constexpr (sizeof(R) == 4) {
        /* dt * sum_l (dmu/dc)_kl D_lm / dx^2 (and / dy^2), from the FP64
         * constants, rounded once */
        const double dtd = (double)D.dt, ix = 1.0 / (double)D.dx, iy = 1.0 / (double)D.dy;
#pragma unroll
        for (int k = 0; k < K; k++)
#pragma unroll
          for (int m = 0; m < K; m++) {
            double sv = 0.0;
#pragma unroll
            for (int l = 0; l < K; l++) sv += D.muc64[p][k][l] * (double)D.Dbulk[p][l][m];
            const float cx = (float)(sv * dtd * ix * ix), cy = (float)(sv * dtd * iy * iy);
            CX2[k][m] = f2pack(cx, cx);
            CY2[k][m] = f2pack(cy, cy);
          }
      }
    }
    BulkStage<R, K> &sg = ws.st[b];
    const int rows = min(TX, g.mx - x0), ncols = min(TY, g.my - y0);
    if (x0 == 0 || x0 + TX >= g.mx || y0 == 0 || y0 + TY >= g.my) {
      /* boundary tile: halo cells outside the domain are copies of interior
       * cells (the box read zeros there) */
      const R *mu = state + off_state + (long long)N * g.plane;
      const int bx0 = D.bc_x[1][0], bx1 = D.bc_x[1][1], by0 = D.bc_y[1][0], by1 = D.bc_y[1][1];
      for (int e = lane; e < 2 * SW + 2 * SH; e += 32) {
        int i, j;
        bool need;
        if (e < 2 * SW) {   /* halo rows x0-1 (top) and x0+rows (bottom) */
          const int side = e >= SW;
          j = e - side * SW;
          i = side ? rows + 1 : 0;
          need = side ? x0 + TX >= g.mx : x0 == 0;
        } else {            /* halo columns y0-1 (left) and y0+ncols (right) */
          const int side = e >= 2 * SW + SH;
          i = e - 2 * SW - side * SH;
          j = side ? ncols + 1 : 0;
          need = side ? y0 + TY >= g.my : y0 == 0;
        }
        int x = x0 - 1 + i, y = y0 - 1 + j;
        if (need && x <= g.mx && y <= g.my) {
          if (x < 0 || x >= g.mx) x = remap(x, g.mx, bx0, bx1);
          if (y < 0 || y >= g.my) y = remap(y, g.my, by0, by1);
          const R *src = mu + (long long)x * g.pitch + y;
#pragma unroll
          for (int k = 0; k < K; k++) sg.M[k][i][j + CO] = ld_step(src + (long long)k * g.plane);
        }
      }
      fence_proxy_async_smem();   /* before a later box overwrites this stage */
      __syncwarp();
    }
    R *phin = next + off_state;
    R *mun = phin + (long long)N * g.plane;
    /* lane 16h + q steps tile rows 4h..4h+3 at columns 2q and 2q+1: stage
     * columns c and c+1 (c = 2q + 1 + CO, so the pair is 16-byte aligned in
     * FP64 and 8-byte aligned in FP32); the y-face between the two cells is
     * computed once, and the x-face below a row is carried to the next */
    const int hh = lane >> 4, qq = lane & 15;
    const int jc = 2 * qq, c = jc + 1 + CO, y = y0 + jc;
    const bool v0 = y < g.my, v1 = y + 1 < g.my;
    const int r0 = 4 * hh, nr = max(0, min(4, rows - r0));
    double acc[SUMS ? NS : 1];
#pragma unroll
    for (int f = 0; f < (SUMS ? NS : 1); f++) acc[f] = 0.0;
    /* the progress sums of one new cell of phase p */
    auto sum_cell = [&](const R (&nm)[K], const double (&dmu)[K]) {
      if constexpr (SUMS) {
        R nph[N];
#pragma unroll
        for (int a = 0; a < N; a++) nph[a] = a == p ? R(1.0) : R(0.0);
#pragma unroll
        for (int k = 0; k < K; k++) acc[N + k] += dmu[k] * dmu[k];
#pragma unroll
        for (int a = 0; a < N; a++) acc[N + K + a] += (double)nph[a];
#pragma unroll
        for (int k = 0; k < K; k++) {
          R comp = R(0.0);
#pragma unroll
          for (int b2 = 0; b2 < N; b2++) comp += c_mu<R, K>(D, nm, b2, k) * h<R, N>(nph, b2);
          acc[2 * N + K + k] += (double)comp;
        }
        bool bad = false;
#pragma unroll
        for (int k = 0; k < K; k++) bad |= !isfinite(nm[k]);
        acc[NS - 1] += bad ? 1.0 : 0.0;
      }
    };
    /* FP64: the new mu of a cell from its old mu and the flux divergences,
     * every term of the K x K matrices (non-DIAG kernels) */
    auto commit_mu = [&](const MatC &mt, const R (&m)[K], const R (&df)[K], R (&nm)[K], double (&dmu)[K]) {
      R cn[K];
#pragma unroll
      for (int k = 0; k < K; k++) {
        R cm = R(0.0);   /* c_mu (functionF_01.h:30-37) */
#pragma unroll
        for (int l = 0; l < K; l++) cm += mt.cmu[k][l] * (m[l] - E[l]);
        cn[k] = cm + dt * (df[k]) - divjat;
      }
#pragma unroll
      for (int k = 0; k < K; k++) {
        R sm = twoA[k] * cn[k] + E[k];   /* Mu (functionF_01.h:19-29) */
#pragma unroll
        for (int l = 0; l < K; l++)
          if (k != l) sm += mt.A[k][l] * cn[l];
        nm[k] = sm;
        dmu[k] = (double)nm[k] - (double)m[k];
      }
    };
    if (v0 && nr > 0) {
      if constexpr (sizeof(R) == 8) {
        /* ---- FP64: the reference's bulk expressions in their order, two cells at a time */
        double2 P[K], FXP[K][K];
        unsigned redo = 0;   /* DIAG: bit 2 rr + e, cell e of row rr to redo with every term */
        R *mq[K];            /* the row's new mu */
#pragma unroll
        for (int k = 0; k < K; k++) mq[k] = mun + k * g.plane + (long long)(x0 + r0) * g.pitch + y;
#pragma unroll
        for (int l = 0; l < K; l++) {
          const double2 pp = *reinterpret_cast<const double2 *>(&sg.M[l][r0][c]);
          P[l] = *reinterpret_cast<const double2 *>(&sg.M[l][r0 + 1][c]);
          const R g0 = bdiv<MUL>(P[l].x - pp.x, idx, ddx, qs), g1 = bdiv<MUL>(P[l].y - pp.y, idx, ddx, qs);
#pragma unroll
          for (int k = 0; k < K; k++)
            if (!DIAG || l == k) FXP[k][l] = make_double2(mc.dm[k][l] * g0, mc.dm[k][l] * g1);
        }
        for (int rr = 0; rr < nr; rr++) {
          const int i = r0 + 1 + rr, x = x0 + i - 1;
          double2 Pn[K];
          R m0[K], m1[K], n0[K], n1[K];
          double d0[K], d1[K];
#pragma unroll
          for (int k = 0; k < K; k++) { m0[k] = P[k].x; m1[k] = P[k].y; }
          if constexpr (DIAG) {
            /* only the diagonal terms: one component at a time */
#pragma unroll
            for (int k = 0; k < K; k++) {
              Pn[k] = *reinterpret_cast<const double2 *>(&sg.M[k][i + 1][c]);
              const R L = sg.M[k][i][c - 1], Rn = sg.M[k][i][c + 2];
              const R dm = mc.dm[k][k];
              const R fx0 = dm * bdiv<MUL>(Pn[k].x - P[k].x, idx, ddx, qs);
              const R fx1 = dm * bdiv<MUL>(Pn[k].y - P[k].y, idx, ddx, qs);
              const R fl = dm * bdiv<MUL>(P[k].x - L, idy, ddy, qs);
              const R fm = dm * bdiv<MUL>(P[k].y - P[k].x, idy, ddy, qs);
              const R fr = dm * bdiv<MUL>(Rn - P[k].y, idy, ddy, qs);
              R a0 = R(0.0), a1 = R(0.0);
              a0 += bdiv<MUL>(fx0 - FXP[k][k].x, idx, ddx, qs);
              a0 += bdiv<MUL>(fm - fl, idy, ddy, qs);
              a1 += bdiv<MUL>(fx1 - FXP[k][k].y, idx, ddx, qs);
              a1 += bdiv<MUL>(fr - fm, idy, ddy, qs);
              FXP[k][k] = make_double2(fx0, fx1);
              /* c_mu, the bulk update and Mu (functionF_01.h:19-37) of the
               * pure phase, diagonal terms only */
              R cm0 = R(0.0), cm1 = R(0.0);
              cm0 += mc.cmu[k][k] * (m0[k] - E[k]);
              cm1 += mc.cmu[k][k] * (m1[k] - E[k]);
              const R cn0 = cm0 + dt * (a0) - divjat, cn1 = cm1 + dt * (a1) - divjat;
              n0[k] = twoA[k] * cn0 + E[k];
              n1[k] = twoA[k] * cn1 + E[k];
              d0[k] = (double)n0[k] - (double)m0[k];
              d1[k] = (double)n1[k] - (double)m1[k];
            }
          } else {
            R gx0[K], gx1[K], gl[K], gm[K], gr[K];
#pragma unroll
            for (int l = 0; l < K; l++) {
              Pn[l] = *reinterpret_cast<const double2 *>(&sg.M[l][i + 1][c]);
              const R L = sg.M[l][i][c - 1], Rn = sg.M[l][i][c + 2];
              gx0[l] = bdiv<MUL>(Pn[l].x - P[l].x, idx, ddx, qs);
              gx1[l] = bdiv<MUL>(Pn[l].y - P[l].y, idx, ddx, qs);
              gl[l] = bdiv<MUL>(P[l].x - L, idy, ddy, qs);
              gm[l] = bdiv<MUL>(P[l].y - P[l].x, idy, ddy, qs);
              gr[l] = bdiv<MUL>(Rn - P[l].y, idy, ddy, qs);
            }
            R df0[K], df1[K];
#pragma unroll
            for (int k = 0; k < K; k++) {
              R a0 = R(0.0), a1 = R(0.0);
#pragma unroll
              for (int l = 0; l < K; l++) {
                const R dm = mc.dm[k][l];
                const R fx0 = dm * gx0[l], fx1 = dm * gx1[l];
                const R fl = dm * gl[l], fm = dm * gm[l], fr = dm * gr[l];
                a0 += bdiv<MUL>(fx0 - FXP[k][l].x, idx, ddx, qs);
                a0 += bdiv<MUL>(fm - fl, idy, ddy, qs);
                a1 += bdiv<MUL>(fx1 - FXP[k][l].y, idx, ddx, qs);
                a1 += bdiv<MUL>(fr - fm, idy, ddy, qs);
                FXP[k][l] = make_double2(fx0, fx1);
              }
              df0[k] = a0;
              df1[k] = a1;
            }
            commit_mu(mc, m0, df0, n0, d0);
            commit_mu(mc, m1, df1, n1, d1);
          }
          /* new extremes, or a value that is not finite */
          bool out = false;
#pragma unroll
          for (int k = 0; k < K; k++) {
            out = out | !(n0[k] <= emax[k]) | !(n0[k] >= emin[k]);
            out = out | (v1 & (!(n1[k] <= emax[k]) | !(n1[k] >= emin[k])));
          }
          const bool srow = stat_row(g, x);   /* the statistics take the cells of their rows */
          if (out) {
            /* a left-out term is +-0 only when the values it multiplies are
             * finite, and they are when every new mu is; otherwise (DIAG) the
             * cell is redone with every term after the rows (its extremes are
             * taken then) */
            bool f0 = true, f1 = v1;
            if constexpr (DIAG) {
#pragma unroll
              for (int k = 0; k < K; k++) { f0 &= fabs(n0[k]) < R(INFINITY); f1 &= fabs(n1[k]) < R(INFINITY); }
              redo |= (f0 ? 0u : 1u) << (2 * rr);
              redo |= (v1 && !f1 ? 2u : 0u) << (2 * rr);
            }
#pragma unroll
            for (int e = 0; e < 2; e++)
              if (srow && (e ? f1 : f0)) {
#pragma unroll
                for (int k = 0; k < K; k++) {
                  const R v = e ? n1[k] : n0[k];
                  if (fabs(v) < R(INFINITY)) {
                    emax[k] = fmax(emax[k], v);
                    emin[k] = fmin(emin[k], v);
                    beaten = true;
                  } else if (v == v && st.ext) {   /* (NaN is ignored) */
                    if (v > R(0.0)) atomicMax(ext_slot(s) + k, ord(v));
                    else atomicMin(ext_slot(s) + K + k, ord(v));
                  }
                }
              }
          }
#pragma unroll
          for (int k = 0; k < K; k++) {
            if (v1) *reinterpret_cast<double2 *>(mq[k]) = make_double2(n0[k], n1[k]);
            else *mq[k] = n0[k];
            mq[k] += g.pitch;
          }
          const long long o = (long long)x * g.pitch + y;
          if (have != p) {
#pragma unroll
            for (int a = 0; a < N; a++) {
              const R v = a == p ? R(1.0) : R(0.0);
              if (v1) *reinterpret_cast<double2 *>(phin + a * g.plane + o) = make_double2(v, v);
              else phin[a * g.plane + o] = v;
            }
          }
          if (SUMS && srow) {
            sum_cell(n0, d0);
            if (v1) sum_cell(n1, d1);
          }
#pragma unroll
          for (int l = 0; l < K; l++) P[l] = Pn[l];
        }
        if constexpr (DIAG) {
          while (redo) {
            const int bit = __ffs(redo) - 1;
            redo &= redo - 1;
            const int i = r0 + 1 + (bit >> 1), cc = c + (bit & 1), x = x0 + i - 1;
            R m[K], nm[K];
            double dmu[K];
#pragma unroll
            for (int k = 0; k < K; k++) m[k] = sg.M[k][i][cc];
            bulk_cell_full_f64<K, MUL>(&sg.M[0][0][0], i, cc, &D, p, m, nm, dmu);
            const long long o = (long long)x * g.pitch + y + (bit & 1);
            const bool srow = stat_row(g, x);
#pragma unroll
            for (int k = 0; k < K; k++) {
              mun[k * g.plane + o] = nm[k];
              if (srow && st.ext && nm[k] == nm[k]) {
                atomicMax(ext_slot(s) + k, ord((double)nm[k]));
                atomicMin(ext_slot(s) + K + k, ord((double)nm[k]));
              }
            }
            if (srow) sum_cell(nm, dmu);
          }
        }
      } else {
        /* ---- FP32: the new mu of a bulk cell is mu + sum_m (CX[k][m] lapx(mu_m)
         * + CY[k][m] lapy(mu_m)) -- the flux divergence of the pure phase's
         * constant D times dt and dmu/dc folded into one coefficient per
         * direction -- in packed f32x2 arithmetic on the cell pair, rounded
         * stochastically by dithering: RN(mu + (s + w ulp(mu))) with w
         * uniform in [-1/2, 1/2) takes the upper neighbour with probability
         * equal to the fraction of the ulp. */
        f2 P[K], DXP[K];
#pragma unroll
        for (int m = 0; m < K; m++) {
          const f2 pp = *reinterpret_cast<const f2 *>(&sg.M[m][r0][c]);
          P[m] = *reinterpret_cast<const f2 *>(&sg.M[m][r0 + 1][c]);
          DXP[m] = f2sub(P[m], pp);
        }
        unsigned rng = mix32(skey ^ ((unsigned)(x0 + r0) * 0x85ebca6bu + (unsigned)y * 0xc2b2ae35u));
        for (int rr = 0; rr < nr; rr++) {
          const int i = r0 + 1 + rr, x = x0 + i - 1;
          f2 Pn[K], LX[K], LY[K];
#pragma unroll
          for (int m = 0; m < K; m++) {
            Pn[m] = *reinterpret_cast<const f2 *>(&sg.M[m][i + 1][c]);
            const float L = (float)sg.M[m][i][c - 1], Rn = (float)sg.M[m][i][c + 2];
            const f2 dxn = f2sub(Pn[m], P[m]);
            LX[m] = f2sub(dxn, DXP[m]);
            DXP[m] = dxn;
            const float px = f2lo(P[m]), py = f2hi(P[m]);
            const f2 o = f2sub(f2pack(px, Rn), f2pack(L, py));   /* (yl, yr) */
            const float ym = __fsub_rn(py, px);
            LY[m] = f2sub(f2pack(ym, f2hi(o)), f2pack(f2lo(o), ym));
          }
          const long long o = (long long)x * g.pitch + y;
          const bool srow = stat_row(g, x);
          R n0[K], n1[K];
          double d0[K], d1[K];
#pragma unroll
          for (int k = 0; k < K; k++) {
            f2 sdm = f2mul(CY2[k][k], LY[k]);
            sdm = f2fma(CX2[k][k], LX[k], sdm);
            if constexpr (!DIAG) {
#pragma unroll
              for (int m = 0; m < K; m++) {
                if (m == k) continue;
                sdm = f2fma(CY2[k][m], LY[m], sdm);
                sdm = f2fma(CX2[k][m], LX[m], sdm);
              }
            }
            const float m0 = f2lo(P[k]), m1 = f2hi(P[k]);
            rng = rng * 1664525u + 1013904223u;
            const float w0 = __uint_as_float(0x3f800000u | (rng >> 9)) - 1.5f;
            rng = rng * 1664525u + 1013904223u;
            const float w1 = __uint_as_float(0x3f800000u | (rng >> 9)) - 1.5f;
            const f2 nm = f2add(P[k], f2fma(f2pack(w0, w1), f2pack(ulpf(m0), ulpf(m1)), sdm));
            n0[k] = f2lo(nm);
            n1[k] = f2hi(nm);
            d0[k] = (double)f2lo(sdm);
            d1[k] = (double)f2hi(sdm);
            if (v1) {
              *reinterpret_cast<f2 *>(mun + k * g.plane + o) = nm;
              if (srow) {
                emax[k] = fmax3f(emax[k], n0[k], n1[k]);
                emin[k] = fmin3f(emin[k], n0[k], n1[k]);
              }
            } else {
              mun[k * g.plane + o] = n0[k];
              if (srow) {
                emax[k] = fmaxf(emax[k], n0[k]);
                emin[k] = fminf(emin[k], n0[k]);
              }
            }
          }
          if (have != p) {
#pragma unroll
            for (int a = 0; a < N; a++) {
              const R v = a == p ? R(1.0) : R(0.0);
              if (v1) *reinterpret_cast<f2 *>(phin + a * g.plane + o) = f2pack(v, v);
              else phin[a * g.plane + o] = v;
            }
          }
          if (srow) {
            sum_cell(n0, d0);
            if (v1) sum_cell(n1, d1);
          }
#pragma unroll
          for (int m = 0; m < K; m++) P[m] = Pn[m];
        }
      }
    }
    if constexpr (SUMS) {
#pragma unroll
      for (int f = 0; f < NS; f++) {
        const double r = warp_sum(acc[f]);
        if (lane == 0) st.partials[(long long)t * NS + f] = r;
      }
    }
    if (lane == 0) flag_out[t] = uniform_flags(p);
    __syncwarp();   /* stage b is refilled by a later issue */
  }
  if (cur_sim >= 0) flush(cur_sim);
}

/* End of a warp's bulk tiles when the same shared memory is used otherwise
 * afterwards: its stage barriers are invalidated (every box it issued has
 * completed or been waited for). */
template <typename R, int K>
__device__ __forceinline__ void bulk_release_warp() {
  BulkWarpSmem<R, K> &ws = reinterpret_cast<BulkWarpSmem<R, K> *>(step_smem_base)[threadIdx.x >> 5];
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int q = 0; q < BulkGeom<R, K>::NST; q++)
      asm volatile("mbarrier.inval.shared::cta.b64 [%0];\n" ::"r"(smem_addr(&ws.bar[q])) : "memory");
  }
  __syncwarp();
}

template <typename R, int N, int K, bool SUMS, bool MUL, bool DIAG>
__global__ void __launch_bounds__(NTI, sizeof(R) == 4 && K == 1 ? 3 : 2) kf_bulk(
    const SimDesc *__restrict__ sims, const Consts<R> *__restrict__ consts, const int4 *blist,
    const __grid_constant__ BoxMaps maps, const TensorMapSlot *__restrict__ tmaps, int buf, const R *state, R *__restrict__ next,
    TileFlags *__restrict__ flag_out, int *__restrict__ ctr, int ndone, const __grid_constant__ StatBufs st) {
  box_begin<1u << MAP_MU, false>(maps, tmaps, buf);
  bulk_tiles<R, N, K, SUMS, MUL, DIAG>(sims, consts, blist, maps, tmaps, buf, state, next, flag_out, ctr, st);
  step_finish(ctr, ndone, st.sweep ? 0 : 1);
}

/* an interface tile's shared memory */
template <typename R, int N, int K>
struct TileSmem32 : ItemCommon<R, N, K> {
  ItemSmem32<R, N, K> t;
};
template <typename R, int N, int K, bool ANISO>
using TileSmem = typename std::conditional<sizeof(R) == 8, ItemSmem<R, N, K, ANISO>, TileSmem32<R, N, K>>::type;

/* What a step kernel needs of a batch of one, as a kernel parameter: constants
 * and layout then come from the constant bank, as operands of the arithmetic.
 * Batches of several simulations read them from global memory (SOLO false). */
template <typename R, bool SOLO>
struct StepArgs {};
template <typename R>
struct StepArgs<R, true> {
  Consts<R> c;
  SimDesc sd;
};
template <typename R, bool SOLO>
__device__ __forceinline__ const Consts<R> &pick_consts(const StepArgs<R, SOLO> &args, const Consts<R> *sc) {
  if constexpr (SOLO) return args.c;
  else return *sc;
}

/* DIRECT: every tile of one simulation on the caller's planes (phi and mu apart,
 * any pitch), without lists, flags, boxes or a progress record: gp_step_noalloc.
 * CTA b takes tiles b, b + grid, ..., the next one's frame on its way by cp.async
 * while one is stepped (planes of any pitch have no tensor map). */
template <typename R, bool DIRECT>
struct DirectArgs {};
template <typename R>
struct DirectArgs<R, true> {
  const R *mu;
  R *mu_next;
  int ntiles, tiles_x;
};

/* Interface tiles of one step: the CTA takes tiles from the interface list
 * until it is empty, the next one's box in flight while one is stepped.  TG: some
 * simulation is non-isothermal.  A box whose bytes do not arrive within the poll
 * limit sets ctr[CTR_ERR]; the CTA then stops taking tiles. */
template <typename R, int N, int K, bool ANISO, bool MUL, bool TG, bool SOLO, bool DIRECT>
__device__ __forceinline__ void general_tiles(const StepArgs<R, SOLO> &args, const DirectArgs<R, DIRECT> &direct,
                                              const SimDesc *__restrict__ sims,
                                              const Consts<R> *__restrict__ consts, const BoxMaps &maps,
                                              const TensorMapSlot *__restrict__ tmaps, int buf,
                                              const R *state, R *__restrict__ next,
                                              TileFlags *__restrict__ flag_out, const int4 *glist,
                                              int *__restrict__ ctr, const StatBufs &st) {
  using CT = typename std::conditional<MUL, ConstsMul<R>, Consts<R>>::type;
  using IG = ItemGeom<R>;
  constexpr int CO = IG::CO, NWI = NTI / 32;
  constexpr unsigned BOX_BYTES = (unsigned)((N + K) * FR * IG::BW * sizeof(R));
  int nlist = 0;
  if constexpr (DIRECT) nlist = direct.ntiles;
  else nlist = *(volatile int *)(ctr + CTR_LIST);
  if (nlist == 0) return;
  const bool late = st.mixed && (blockIdx.x & 1);   /* after its bulk tiles */
  const int first = late ? -1 : (st.mixed ? blockIdx.x >> 1 : blockIdx.x);
  const int nfirst = st.mixed ? (gridDim.x + 1) >> 1 : gridDim.x;
  using SM = TileSmem<R, N, K, ANISO>;
  SM &sm = *reinterpret_cast<SM *>(step_smem_base);
  __shared__ __align__(16) unsigned char sc_raw[SOLO ? 16 : sizeof(Consts<R>)];
  Consts<R> *const scp = reinterpret_cast<Consts<R> *>(sc_raw);
  const CT &D = static_cast<const CT &>(pick_consts<R, SOLO>(args, scp));
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  auto entry = [&](int i) {
    /* (fits: the size limit on padded planes leaves at most 8192 rows of tiles) */
    if constexpr (DIRECT) return make_int4(i, 0, ((i / direct.tiles_x) << 16) | (i % direct.tiles_x), 0);
    else return ld_step(glist + i);
  };
  const TensorMapSlot *ready = nullptr;
  /* thread 0: note an entry in slot c and start its box */
  auto issue = [&](const int4 &en, int c) {
    sm.ent[c] = en;
    if (!DIRECT && en.x >= 0 && en.w) {
      const unsigned bar = smem_addr(&sm.bar[c]);
      mbar_expect_tx(bar, BOX_BYTES + st.tma_extra[MAP_ALL]);
      tma_load_3d(smem_addr(&sm.F[c]), box_map(maps, tmaps, en.y, buf, MAP_ALL, ready),
                  (en.z & 0xffff) * TY - 2 - CO, (en.z >> 16) * TX - 2, 0, bar);
    }
  };
  if (tid == 0) {
    mbar_init(smem_addr(&sm.bar[0]), 1);
    mbar_init(smem_addr(&sm.bar[1]), 1);
    fence_barrier_init();
    fence_proxy_async_smem();
    if constexpr (sizeof(R) == 8) sm.n_test = sm.n_act = sm.n_task = sm.n_extra = sm.n_j = 0;
    else sm.t.nlist = sm.t.nflist = 0;
    /* the CTAs that begin with interface tiles own the first entries */
    const int i = DIRECT || first >= 0 ? first : nfirst + atomicAdd(ctr + CTR_HEAD, 1);
    issue(i < nlist ? entry(i) : make_int4(-1, 0, 0, 0), 0);
  }
  int cur_sim = -1;
  unsigned parity = 0;   /* bit c: the phase of slot c's barrier its next box completes */
  Grid g = {};
  long long off_state = 0;
  const double *tpf = nullptr, *tcc = nullptr;
  /* DIRECT: the frame of tile t into slot c, every thread its cells */
  auto fetch = [&](int t, int c) {
    if constexpr (DIRECT) {
      const Grid &gd = args.sd.g;
      const int x0 = t / direct.tiles_x * TX, y0 = (t - t / direct.tiles_x * direct.tiles_x) * TY;
      const bool inside = x0 >= 2 && x0 + TX + 2 <= gd.mx && y0 >= 2 && y0 + TY + 2 <= gd.my;
      for (int q = tid; q < FR * FC; q += NTI) {
        const int i = q / FC, j = q - i * FC;
        int x = x0 - 2 + i, y = y0 - 2 + j, xm = x, ym = y;
        unsigned np = 8, nm = 8;
        if (!inside) {
          /* the cells after the boundary remap of phi and mu; zeros where no needed
           * cell lies (phi: [-2, m+1], mu: [-1, m]) */
          const bool need = x < gd.mx + 2 && y < gd.my + 2;
          const bool needm = x >= -1 && x < gd.mx + 1 && y >= -1 && y < gd.my + 1;
          np = need ? 8 : 0;
          nm = needm ? 8 : 0;
          xm = needm ? remap(x, gd.mx, D.bc_x[1][0], D.bc_x[1][1]) : 0;
          ym = needm ? remap(y, gd.my, D.bc_y[1][0], D.bc_y[1][1]) : 0;
          x = need ? remap(x, gd.mx, D.bc_x[0][0], D.bc_x[0][1]) : 0;
          y = need ? remap(y, gd.my, D.bc_y[0][0], D.bc_y[0][1]) : 0;
        }
        const R *cell = state + plane_offset(gd, x, y), *cellm = direct.mu + plane_offset(gd, xm, ym);
#pragma unroll
        for (int a = 0; a < N; a++) cp_async8(&sm.F[c][a][i][j + CO], cell + a * gd.plane, np);
#pragma unroll
        for (int k = 0; k < K; k++) cp_async8(&sm.F[c][N + k][i][j + CO], cellm + k * gd.plane, nm);
      }
    }
  };
  if (DIRECT) fetch(first, 0);
  __syncthreads();
#pragma unroll 1
  for (int cur = 0;; cur ^= 1) {
    const int4 en = sm.ent[cur];
    if (en.x < 0) break;
    const int t = en.x, s = SOLO ? 0 : en.y, x0 = (en.z >> 16) * TX, y0 = (en.z & 0xffff) * TY;
    int nxt = 0;
    if (DIRECT) nxt = t + (int)gridDim.x;
    else if (tid == 0) nxt = nfirst + atomicAdd(ctr + CTR_HEAD, 1);   /* used after the next barrier */
    if (s != cur_sim) {
      cur_sim = s;
      if constexpr (!SOLO) {
        const int *src = reinterpret_cast<const int *>(consts + s);
        int *dst = reinterpret_cast<int *>(scp);
        for (int w = tid; w < (int)(sizeof(Consts<R>) / sizeof(int)); w += NTI) dst[w] = __ldg(src + w);
      }
      if (lane < 2 * (N + K)) {
        const long long o = st.ext ? *(volatile long long *)(st.ext + (long long)s * (2 * (N + K)) + lane) : 0;
        sm.ext[wid][lane] = __longlong_as_double(o < 0 ? o ^ 0x7fffffffffffffffLL : o);
      }
      if constexpr (SOLO) {
        g = args.sd.g;
        off_state = args.sd.off_state;
      } else {
        const SimDesc sd = sims[s];
        g = sd.g;
        off_state = sd.off_state;
        if (TG && st.trows) {
          tpf = st.trows + sd.off_T;
          tcc = tpf + (g.my + 6);
        }
      }
      __syncthreads();
    }
    R(&F)[N + K][FR][IG::BW] = sm.F[cur];
    bool ok = true;
    if constexpr (DIRECT) {
      cp_async_wait();
      __syncthreads();   /* everyone's cells of this frame; the other slot was last read a tile ago */
      if (nxt < nlist) fetch(nxt, cur ^ 1);
    } else if (en.w) {
      ok = mbar_wait(smem_addr(&sm.bar[cur]), (parity >> cur) & 1u, st.mbar_tries[MAP_ALL]);
      parity ^= 1u << cur;
    } else {
      /* rows and columns of the frame after the boundary remap of phi and mu;
       * -1 where no needed cell lies (phi: [-2, m+1], mu: [-1, m]) */
      if (tid < 2 * (FR + FC)) {
        const int f = tid / (FR + FC), u = tid - f * (FR + FC), reach = 2 - f;
        if (u < FR) {
          const int x = x0 - 2 + u;
          sm.row[f][u] = (x >= -reach && x < g.mx + reach) ? remap(x, g.mx, D.bc_x[f][0], D.bc_x[f][1]) : -1;
        } else {
          const int y = y0 - 2 + (u - FR);
          sm.col[f][u - FR] = (y >= -reach && y < g.my + reach) ? remap(y, g.my, D.bc_y[f][0], D.bc_y[f][1]) : -1;
        }
      }
      __syncthreads();
      const R *src = state + off_state, *srcm = src + N * g.plane;
      for (int q = tid; q < FR * FC; q += NTI) {
        const int i = q / FC, j = q - i * FC;
        const int r = sm.row[0][i], c = sm.col[0][j], rm = sm.row[1][i], cm = sm.col[1][j];
        R v[N + K];
#pragma unroll
        for (int f = 0; f < N + K; f++) v[f] = R(0.0);
        if (r >= 0 && c >= 0) {
          const R *cell = src + plane_offset(g, r, c);
#pragma unroll
          for (int a = 0; a < N; a++) v[a] = ld_step(cell + a * g.plane);
        }
        if (rm >= 0 && cm >= 0) {
          const R *cell = srcm + plane_offset(g, rm, cm);
#pragma unroll
          for (int k = 0; k < K; k++) v[N + k] = ld_step(cell + k * g.plane);
        }
#pragma unroll
        for (int f = 0; f < N + K; f++) F[f][i][j + CO] = v[f];
      }
      fence_proxy_async_smem();   /* before a later box overwrites this slot */
      __syncthreads();
    }

    const int tx = wid, ty = lane, x = x0 + tx, y = y0 + ty;
    const bool valid = x < g.mx && y < g.my;
    R dp[N], nph[N], nm[K];
    double dmu[K];
    const double Tc = (TG && D.tgrad && valid) ? ld_step(tcc + y + 3) : 0.0;
    if constexpr (sizeof(R) == 4) {
      if (!__syncthreads_and(ok)) {
        if (tid == 0) atomicExch(ctr + CTR_ERR, 1);
        break;   /* no other box is in flight */
      }
      int4 nent = make_int4(-1, 0, 0, 0);
      if (tid == 0 && nxt < nlist) nent = entry(nxt);
      tile32<R, N, K, ANISO>(D, g, F, x0, y0, st, sm.t, tpf, tcc, dp, nph, nm, dmu, [&]() {
        if (tid == 0) issue(nent, cur ^ 1);   /* the other slot was last read a tile ago */
      });
    } else {
    /* ---- ring cells, a warp per row and one for the last two columns: a constant
     * 5-point stencil has no active phase (delta-phi is 0, or the projection's clamp
     * of a negative phi), the others are listed; D; whether the fields are of
     * ordinary size (left-out terms are then +-0) */
    bool tame = D.quick_span != 0;
    for (int rt = wid; rt < RR + 1; rt += NWI) {
      const int ri = rt < RR ? rt : lane >> 1, rj = rt < RR ? lane : 32 + (lane & 1);
      const bool in = rt < RR || lane < 2 * RR;
      const int i = ri + 1, j = rj + 1, e = RI(ri, rj);
      const bool vd = in && (x0 - 1 + ri <= g.mx) && (y0 - 1 + rj <= g.my);
      bool nu = false;
      R p[N];
#pragma unroll
      for (int a = 0; a < N; a++) p[a] = R(0.0);
      if (vd) {
#pragma unroll
        for (int a = 0; a < N; a++) {
          p[a] = F[a][i][j + CO];
          /* bitwise, not short-circuit: branches here cost more than the comparisons */
          tame = tame & (fabs(p[a]) < R(PHI_TAME));
          nu = nu | (F[a][i + 1][j + CO] != p[a]) | (F[a][i - 1][j + CO] != p[a]) | (F[a][i][j + 1 + CO] != p[a]) |
               (F[a][i][j - 1 + CO] != p[a]);
        }
#pragma unroll
        for (int k = 0; k < K; k++) tame = tame & (fabs(F[N + k][i][j + CO]) < R(MU_TAME));
        /* (a constant stencil between phases is listed too, for its anti-trapping weights) */
#pragma unroll
        for (int a = 0; a < N - 1; a++) nu = nu | ((p[a] != R(0.0)) & (p[a] != R(1.0)));
      }
      if (in) {
        if (!nu) {
          sm.ACT[e] = 0;
#pragma unroll
          for (int a = 0; a < N; a++) {
            R d = R(0.0);
            if ((p[a] + d) < R(0.0)) d += fabs(d + p[a]);
            sm.DP[a][e] = d;
          }
        }
#pragma unroll
        for (int k = 0; k < K; k++)
#pragma unroll
          for (int l = 0; l < K; l++) {
            if (k != l && st.diag) continue;
            R v = R(0.0);
#pragma unroll
            for (int b = 0; b < N; b++)
#pragma unroll
              for (int n = 0; n < K; n++)
                if (n == k || !st.diag) v += D.DC[b][k][l][n] * p[b];
            sm.DD[k][l][e] = v;
          }
      }
      const unsigned m = __ballot_sync(0xffffffffu, nu);
      if (lane == 0) {
        if (rt < RR) sm.NU[rt] = m;
        else sm.NUX = m;
      }
      if (m) {
        int b = 0;
        if (lane == 0) b = atomicAdd(&sm.n_test, __popc(m));
        b = __shfl_sync(0xffffffffu, b, 0);
        if (nu) sm.TEST[b + __popc(m & ((1u << lane) - 1u))] = (short)e;
      }
    }
    {
      /* the phi of the frame around the ring, by warps that had one row above */
      const int q = tid - (RR + 1 - NWI) * 32;
      constexpr int TOP = 2 * FC, ALL = TOP + 2 * (FR - 2);
      if (q >= 0 && q < ALL) {
        const int i = q < TOP ? (q < FC ? 0 : FR - 1) : 1 + ((q - TOP) >> 1);
        const int j = q < TOP ? (q < FC ? q : q - FC) : ((q - TOP) & 1) * (FC - 1);
#pragma unroll
        for (int a = 0; a < N; a++) tame = tame & (fabs(F[a][i][j + CO]) < R(PHI_TAME));
      }
    }
    tame = __syncthreads_and(ok && tame);
    if (!tame) {
      if (!__syncthreads_and(ok)) {
        if (tid == 0) atomicExch(ctr + CTR_ERR, 1);
        break;   /* no other box is in flight */
      }
      if (K > 1 && st.diag) {   /* the off-diagonal D left out above */
        for (int e = tid; e < RS; e += NTI) {
          R p[N];
#pragma unroll
          for (int a = 0; a < N; a++) p[a] = F[a][e / RC + 1][e % RC + 1 + CO];
#pragma unroll
          for (int k = 0; k < K; k++)
#pragma unroll
            for (int l = 0; l < K; l++) sm.DD[k][l][e] = Dcell<R, N, K>(D, p, k, l);
        }
        __syncthreads();
      }
    }
    const bool dg = st.diag && tame;
    int4 nent = make_int4(-1, 0, 0, 0);
    if (tid == 0 && nxt < nlist) nent = entry(nxt);

    /* a tile without a listed cell has no active phase and no current */
    const bool listed = sm.n_test != 0;
    if (!listed) {
      if (tid == 0) issue(nent, cur ^ 1);   /* the other slot was last read a tile ago */
    } else {
    /* ---- listed cells: active phases */
    const int ntest = sm.n_test;
    for (int q0 = 32 * wid; q0 < ntest; q0 += NTI) {
      const int q = q0 + lane;
      unsigned mask = 0;
      int e = 0;
      if (q < ntest) {
        e = sm.TEST[q];
        const int ri = e / RC, rj = e - ri * RC, i = ri + 1, j = rj + 1;
        R p[N];
#pragma unroll
        for (int a = 0; a < N; a++) {
          p[a] = F[a][i][j + CO];
          const R xp = F[a][i + 1][j + CO], xm = F[a][i - 1][j + CO], yp = F[a][i][j + 1 + CO],
                  ym = F[a][i][j - 1 + CO];
          /* a phase that is zero on the stencil is not active */
          if (N > 2 && ((p[a] == R(0.0)) & (xp == R(0.0)) & (xm == R(0.0)) & (yp == R(0.0)) & (ym == R(0.0)))) continue;
          R dv = divx(divx(xp - p[a], D) - divx(p[a] - xm, D), D);
          dv += divy(divy(yp - p[a], D) - divy(p[a] - ym, D), D);
          if (fabs(dv) > R(0.0)) mask |= 1u << a;
        }
        sm.ACT[e] = (unsigned char)mask;
        if (!mask) {
#pragma unroll
          for (int a = 0; a < N; a++) {
            R d = R(0.0);
            if ((p[a] + d) < R(0.0)) d += fabs(d + p[a]);
            sm.DP[a][e] = d;
          }
        }
        if (D.obstacle) {
          /* a solid between 0 and 1 that is not active (the active ones' weights come with the lambdas) */
#pragma unroll 1
          for (int a = 0; a < N - 1; a++) {
            const R pa = F[a][i][j + CO];
            if (!((mask >> a) & 1u) && pa * (R(1.0) - pa) > R(0.0)) sm.SP[a][e] = item_sphi<R, N, K>(F, i, j, a);
          }
        }
      }
      const unsigned m = __ballot_sync(0xffffffffu, mask != 0);
      if (m) {
        unsigned ma[N];
        int nt = 0, b = 0, bt = 0;
#pragma unroll
        for (int a = 0; a < N; a++) {
          ma[a] = __ballot_sync(0xffffffffu, (mask >> a) & 1u);
          nt += __popc(ma[a]);
        }
        if (lane == 0) {
          b = atomicAdd(&sm.n_act, __popc(m));
          bt = atomicAdd(&sm.n_task, nt);
        }
        b = __shfl_sync(0xffffffffu, b, 0);
        bt = __shfl_sync(0xffffffffu, bt, 0);
        const unsigned below = (1u << lane) - 1u;
        if (mask) sm.LIST[b + __popc(m & below)] = (short)e;
#pragma unroll
        for (int a = 0; a < N; a++) {
          if ((mask >> a) & 1u) sm.TASK[bt + __popc(ma[a] & below)] = (short)(e | (a << 10));
          bt += __popc(ma[a]);
        }
      }
    }
    /* ---- faces next to a cell with a varying stencil, a warp per row of faces */
    for (int q = wid; q < 2 * TX + 1; q += NWI) {
      const int r = q <= TX ? q : q - TX;   /* ring row; x-faces lie between it and the next one */
      const unsigned long long a = sm.NU[r] | (unsigned long long)((sm.NUX >> (2 * r)) & 3u) << 32;
      unsigned long long w;
      if (q <= TX) {
        const unsigned long long c = sm.NU[r + 1] | (unsigned long long)((sm.NUX >> (2 * r + 2)) & 3u) << 32;
        w = ((a | c) >> 1) & 0xffffffffull;
      } else {
        w = (a | (a >> 1)) & 0x1ffffffffull;
      }
      const unsigned lo = (unsigned)w;
      int b = 0;
      if (lane == 0) {
        sm.JW[q] = w;
        if (w) b = atomicAdd(&sm.n_j, __popcll(w));
      }
      if (w) {
        b = __shfl_sync(0xffffffffu, b, 0);
        const int f = q <= TX ? q * TY : JXF + (q - TX - 1) * (TY + 1);
        if ((lo >> lane) & 1u) sm.JLIST[b + __popc(lo & ((1u << lane) - 1u))] = (short)(f + lane);
        if (lane == 0 && (w >> 32)) sm.JLIST[b + __popc(lo)] = (short)(f + TY);
      }
    }
    __syncthreads();
    const int nact = sm.n_act, ntask = sm.n_task;
    if (tid == 0) issue(nent, cur ^ 1);   /* the other slot was last read a tile ago */
    if (ANISO && nact > 0) {
      /* the faces of active cells, each once: forward x and right y of every
       * cell, and the backward ones whose other cell is not active */
      for (int q0 = 32 * wid; q0 < nact; q0 += NTI) {
        const int q = q0 + lane;
        bool bx_ = false, by_ = false;
        int ri = 0, rj = 0;
        if (q < nact) {
          const int e = sm.LIST[q];
          ri = e / RC;
          rj = e - ri * RC;
          sm.FLIST[q] = (short)((ri + 1) * RC + rj);
          sm.FLIST[nact + q] = (short)(IXF + ri * (TY + 3) + rj + 1);
          bx_ = ri == 0 || !sm.ACT[e - RC];
          by_ = rj == 0 || !sm.ACT[e - 1];
        }
        const unsigned mx_ = __ballot_sync(0xffffffffu, bx_), my_ = __ballot_sync(0xffffffffu, by_);
        int b = 0;
        if (lane == 0) b = atomicAdd(&sm.n_extra, __popc(mx_) + __popc(my_));
        b = 2 * nact + __shfl_sync(0xffffffffu, b, 0);
        const unsigned below = (1u << lane) - 1u;
        if (bx_) sm.FLIST[b + __popc(mx_ & below)] = (short)(ri * RC + rj);
        if (by_) sm.FLIST[b + __popc(mx_) + __popc(my_ & below)] = (short)(IXF + ri * (TY + 3) + rj);
      }
      __syncthreads();
      const int nf = 2 * nact + sm.n_extra;
      for (int q = tid; q < nf; q += NTI) item_face<R, N, K, ANISO>(D, F, sm, sm.FLIST[q], tame);
      __syncthreads();
    }
    {
      /* lambda of each active (cell, phase), and on the threads after them the
       * anti-trapping weights of the active cells' solids */
      const int t32 = (ntask + 31) & ~31, all = D.obstacle ? t32 + nact : ntask;
      for (int q = tid; q < all; q += NTI) {
        if (q < ntask) {
          const int v = sm.TASK[q], e = v & 1023;
          item_lambda<R, N, K, ANISO, TG>(D, F, sm, e, v >> 10, tame, dg,
                                          TG && D.tgrad ? ld_step(tpf + y0 - 1 + e % RC + 3) : 0.0);
        } else if (q >= t32) {
          const int e = sm.LIST[q - t32], ri = e / RC, rj = e - ri * RC;
          const unsigned act = sm.ACT[e];
#pragma unroll 1
          for (int a = 0; a < N - 1; a++) {
            const R p = F[a][ri + 1][rj + 1 + CO];
            if (((act >> a) & 1u) && p * (R(1.0) - p) > R(0.0)) sm.SP[a][e] = item_sphi<R, N, K>(F, ri + 1, rj + 1, a);
          }
        }
      }
    }
    __syncthreads();
    const int nj = sm.n_j;
    for (int q = tid; q < nact; q += NTI) item_dphi<R, N, K, ANISO>(D, F, sm, sm.LIST[q]);
    __syncthreads();
    if (tid == 0) sm.n_test = sm.n_act = sm.n_task = sm.n_extra = sm.n_j = 0;   /* for the next tile */
    if (nj > 0) {
      for (int q = tid; q < nj; q += NTI)
        item_current<R, N, K, ANISO, TG>(D, F, sm, sm.JLIST[q], y0, g.my, dg, tcc);
      __syncthreads();
    }
    }
    if (st.dphi_out) {
      /* the adjoint's tape: the delta-phi of the tile and of its ring cells
       * (the domain's ring included), as the reverse sweep reads it */
      for (int e = tid; e < RS; e += NTI) {
        const int x = x0 - 1 + e / RC, y = y0 - 1 + e % RC;
        if (x <= g.mx && y <= g.my) {
#pragma unroll
          for (int a = 0; a < N; a++)
            st.dphi_out[a * g.dplane + (long long)(x + 1) * g.dpitch + (y + 1)] = (double)sm.DP[a][e];
        }
      }
    }

    /* ---- per cell: mu update, phi commit */
    if (valid) {
      R ph[N], m[K];
#pragma unroll
      for (int a = 0; a < N; a++) {
        ph[a] = F[a][tx + 2][ty + 2 + CO];
        dp[a] = sm.DP[a][RI(tx + 1, ty + 1)];
      }
#pragma unroll
      for (int k = 0; k < K; k++) m[k] = F[N + k][tx + 2][ty + 2 + CO];
      item_commit<R, N, K, ANISO, TG>(D, F, sm, tx, ty, x, y, tame, dg, listed, ph, dp, m, nph, nm, dmu, Tc);
    }
    }
    int oh = -1;
    if (valid) {
      R *out = next + off_state + (long long)x * g.pitch + y, *outm = out + N * g.plane;
      if constexpr (DIRECT) outm = direct.mu_next + (long long)x * g.pitch + y;
#pragma unroll
      for (int a = 0; a < N; a++) out[a * g.plane] = nph[a];
#pragma unroll
      for (int k = 0; k < K; k++) outm[k * g.plane] = nm[k];
      oh = one_hot<R, N>(nph);
    } else {
#pragma unroll
      for (int a = 0; a < N; a++) nph[a] = R(0.0);
#pragma unroll
      for (int k = 0; k < K; k++) nm[k] = R(0.0);
    }
    if (st.ext && stat_row(g, x)) item_extremes<R, N, K>(sm.ext[wid], valid, nph, nm, st, s);
    {
      const unsigned b = row_flag_bits<N>(valid, oh);
      if (lane == 0) sm.fm[cur][wid] = b;
    }
    if (st.want_sums) item_sums<R, N, K, TG>(D, valid && stat_row(g, x), nph, nm, dp, dmu, st, t, Tc);
    __syncthreads();   /* the tile's shared memory is free, its rows' flag bits are written */
    if (!DIRECT && tid == 32) flag_out[t] = flags_of_rows(sm.fm[cur]);
  }
  __syncthreads();
  if (tid == 0) {
    asm volatile("mbarrier.inval.shared::cta.b64 [%0];\n" ::"r"(smem_addr(&sm.bar[0])) : "memory");
    asm volatile("mbarrier.inval.shared::cta.b64 [%0];\n" ::"r"(smem_addr(&sm.bar[1])) : "memory");
  }
  __syncthreads();
}

/* The interface tiles in a kernel: inlined in FP64; in FP32 one copy that every
 * kernel calls, so that its fused multiply-adds are the same in all of them. */
template <int N, int K, bool ANISO, bool TG>
__device__ __noinline__ void general_tiles_f32(const SimDesc *__restrict__ sims, const Consts<float> *__restrict__ consts,
                                               const BoxMaps &maps, const TensorMapSlot *__restrict__ tmaps, int buf,
                                               const float *state, float *__restrict__ next,
                                               TileFlags *__restrict__ flag_out, const int4 *glist,
                                               int *__restrict__ ctr, const StatBufs st) {
  general_tiles<float, N, K, ANISO, true, TG, false, false>(StepArgs<float, false>{}, DirectArgs<float, false>{}, sims, consts, maps, tmaps, buf,
                                                     state, next, flag_out, glist, ctr, st);
}
template <typename R, int N, int K, bool ANISO, bool MUL, bool TG, bool SOLO>
__device__ __forceinline__ void step_general(const StepArgs<R, SOLO> &args, const SimDesc *__restrict__ sims,
                                             const Consts<R> *__restrict__ consts, const BoxMaps &maps,
                                             const TensorMapSlot *__restrict__ tmaps, int buf,
                                             const R *state, R *__restrict__ next,
                                             TileFlags *__restrict__ flag_out, const int4 *glist,
                                             int *__restrict__ ctr, const StatBufs &st) {
  if constexpr (sizeof(R) == 8)
    general_tiles<R, N, K, ANISO, MUL, TG, SOLO, false>(args, DirectArgs<R, false>{}, sims, consts, maps, tmaps, buf,
                                                        state, next, flag_out, glist, ctr, st);
  else
    general_tiles_f32<N, K, ANISO, TG>(sims, consts, maps, tmaps, buf, state, next, flag_out, glist, ctr, st);
}

/* CTAs of the interface code an SM holds: what its shared memory leaves, at most two (128 registers a thread) */
template <typename R, int N, int K, bool ANISO>
constexpr int item_ctas() {
  constexpr size_t need = sizeof(TileSmem<R, N, K, ANISO>) + 128 + sizeof(Consts<R>) + 2048;
  constexpr int n = (int)(228 * 1024 / need);
  return n < 1 ? 1 : (n > 2 ? 2 : n);
}

template <typename R, int N, int K, bool ANISO, bool MUL, bool TG, bool SOLO>
__global__ void __launch_bounds__(NTI, item_ctas<R, N, K, ANISO>()) kf_general(
    const __grid_constant__ StepArgs<R, SOLO> args, const SimDesc *__restrict__ sims,
    const Consts<R> *__restrict__ consts, const __grid_constant__ BoxMaps maps,
    const TensorMapSlot *__restrict__ tmaps, int buf, const R *state, R *__restrict__ next,
    TileFlags *__restrict__ flag_out, const int4 *glist, int *__restrict__ ctr, int ndone, const __grid_constant__ StatBufs st) {
  box_begin<1u << MAP_ALL, SOLO>(maps, tmaps, buf);
  step_general<R, N, K, ANISO, MUL, TG, SOLO>(args, sims, consts, maps, tmaps, buf, state, next, flag_out, glist, ctr,
                                                 st);
  step_finish(ctr, ndone, 1);
}

/* One step of one simulation on the caller's planes (gp_step_noalloc).  On a grid of
 * many tiles, most of them without an interface, the latency of a tile bounds it:
 * hence the next frame on its way and the short path of a tile without a listed cell.
 * A CTA takes two tiles where there are more tiles than resident CTAs, so that a free
 * SM takes the next two: with all tiles dealt out at the start the CTA with the most
 * interface tiles ended late (1000x300: 45 us; two tiles 29, one tile 31), and one
 * tile per CTA has no next frame (1440x1400, one seed: 88 us, two tiles 78).  Binary
 * anisotropic 1440x1400 with 20 seeds: two passes of small CTAs over a delta-phi array
 * 111 us, one launch without all this 160 us, with it 93 us; three-phase ternary
 * 1160x1130: 161, 125 and 85 us. */
constexpr int NOALLOC_TILES = 2;
template <typename R, int N, int K, bool ANISO, bool MUL>
__global__ void __launch_bounds__(NTI, item_ctas<R, N, K, ANISO>()) kn_step(
    const __grid_constant__ StepArgs<R, true> args, const __grid_constant__ DirectArgs<R, true> direct,
    const R *__restrict__ phi, R *__restrict__ phi_next, const __grid_constant__ StatBufs st) {
  general_tiles<R, N, K, ANISO, MUL, false, true, true>(args, direct, nullptr, nullptr, BoxMaps{}, nullptr, 0, phi,
                                                        phi_next, nullptr, nullptr, nullptr, st);
}

/* One step in one persistent launch: each CTA takes interface tiles while
 * the interface list lasts, then its warps take bulk tiles, so the two kinds
 * of work share the SMs and the step ends with one tail instead of two.  In a
 * mixed shape the odd CTAs take them the other way round: the two kinds of work
 * then share every SM from the start of the step. */
template <typename R, int N, int K, bool ANISO, bool MUL, bool TG, bool SOLO, bool DIAG>
__global__ void __launch_bounds__(NTI, item_ctas<R, N, K, ANISO>()) kf_step(
    const __grid_constant__ StepArgs<R, SOLO> args, const SimDesc *__restrict__ sims,
    const Consts<R> *__restrict__ consts, const int4 *blist, const int4 *glist, const __grid_constant__ BoxMaps maps,
    const TensorMapSlot *__restrict__ tmaps, int buf, const R *state, R *__restrict__ next,
    TileFlags *__restrict__ flag_out, int *__restrict__ ctr, int ndone, const __grid_constant__ StatBufs st) {
  box_begin<1u << MAP_MU | 1u << MAP_ALL, SOLO>(maps, tmaps, buf);
  const int bulk_pass = st.mixed && (blockIdx.x & 1) ? 0 : 1;
#pragma unroll 1
  for (int pass = 0; pass < 2; pass++) {
    if (pass == bulk_pass) {
      bulk_tiles<R, N, K, false, MUL, DIAG>(sims, consts, blist, maps, tmaps, buf, state, next, flag_out, ctr, st);
      bulk_release_warp<R, K>();
    } else {
      step_general<R, N, K, ANISO, MUL, TG, SOLO>(args, sims, consts, maps, tmaps, buf, state, next, flag_out, glist,
                                                   ctr, st);
    }
    __syncthreads();   /* the pass's shared memory becomes the next one's */
  }
  step_finish(ctr, ndone, 1);
}

/* Per simulation, the moving-frame state the temperature rows need: the
 * offset of the frame, and after a shift the offset and distance the
 * shifted temperature field was laid down with (consumed by the next step). */
struct SimDyn {
  long long shift_off;   /* shift_OFFSET (microsim_gp.c:122) */
  long long shift_T;     /* the offset of the temperature field being shifted */
  int dlast;             /* its shift distance */
  int fresh;             /* a shift happened at the end of the last step */
  int pos;               /* MAX_INTERFACE_POS of the last check */
  int pad;
};

/* The temperature of every ghosted column y of a non-isothermal simulation
 * during the coming step, one CTA per simulation.  The reference's field is
 * temp_bottom + y*GRADIENT (apply_temperature_gradientY, Temperature_gradient.h:4-29),
 * laid down after each step with the step's BASE_POS (microsim_gp.c:108-113;
 * at t = 0 without the velocity term, :77-82) and copied into the ghost
 * columns only by the next boundary copy: the phase-field pass of step t+1
 * reads the field as laid down (as copied at t = 0, where the start-up copy
 * came after it), the concentration pass reads it copied.  After a moving-
 * frame shift the field holds the shifted columns (shift.h:20) until the
 * next step lays it down again.  Rows: [0, MESH_Y+6) as the phase-field pass
 * reads them, then [0, MESH_Y+6) as the concentration pass reads them. */
template <typename R>
__global__ void __launch_bounds__(128) kt_rows(const SimDesc *__restrict__ sims, const Consts<R> *__restrict__ consts,
                                               const int *__restrict__ ctr, SimDyn *__restrict__ dyn,
                                               double *__restrict__ trows) {
  const int s = blockIdx.x;
  const Consts<R> &D = consts[s];
  if (!D.tgrad) return;
  const SimDesc sd = sims[s];
  const int my = sd.g.my, ry = my + 6;
  const long t0 = (long)(unsigned)ctr[CTR_STEP];
  const SimDyn dd = dyn[s];
  const long long shT = dd.fresh ? dd.shift_T : dd.shift_off;
  const long d = dd.fresh ? dd.dlast : 0;
  double base_pos;
  if (t0 == 0) base_pos = (D.tg_off / D.dy64) - (double)shT;
  else base_pos = (D.tg_off / D.dy64) - (double)shT + ((D.tg_vel / D.dy64) * ((double)t0 * D.dt64));
  const double grad = (D.tg_dT) * D.dy64 / (D.tg_dist);
  const double tb = D.tg_base - base_pos * grad;
  double *tpf = trows + sd.off_T, *tcc = tpf + ry;
  for (int y = threadIdx.x; y < ry; y += blockDim.x) {
    /* the column a ghost column is a copy of (T's own boundary types; other
     * types copy nothing) */
    int yr = y;
    if (y < 3 && (D.bc_t[0] == GP_BC_NEUMANN || D.bc_t[0] == GP_BC_PERIODIC))
      yr = remap(y - 3, my, D.bc_t[0], D.bc_t[1]) + 3;
    else if (y >= my + 3 && (D.bc_t[1] == GP_BC_NEUMANN || D.bc_t[1] == GP_BC_PERIODIC))
      yr = remap(y - 3, my, D.bc_t[0], D.bc_t[1]) + 3;
    const double laid = y <= ry - 1 - d ? tb + (double)(y + d) * grad : tb + (double)y * grad;
    const double copied = yr <= ry - 1 - d ? tb + (double)(yr + d) * grad : tb + (double)yr * grad;
    tcc[y] = copied;
    tpf[y] = t0 == 0 ? copied : laid;
  }
  __syncthreads();
  if (threadIdx.x == 0 && dd.fresh) dyn[s].fresh = 0;
}

/* ---- moving frame (Shift = 1) --------------------------------------------
 * Every 100 steps the reference finds MAX_INTERFACE_POS, the largest column y
 * where the liquid crosses one half upwards (check_SHIFT, shift.h:47-65, run
 * over the rows its concentration sweep has just updated), and when it is
 * past Shiftj moves every row down by d = MAX_INTERFACE_POS - Shiftj cells,
 * the top d cells becoming liquid at cfill (apply_shiftY, shift.h:4-45;
 * microsim_gp.c:115-123).  Columns are ghosted indices (interior y + 3). */

/* MAX_INTERFACE_POS over the interior (pairs of interior columns y-1, y),
 * one CTA per tile, atomic max into pos[simulation] */
template <typename R, int N>
__global__ void __launch_bounds__(NT) ks_pos(const SimDesc *__restrict__ sims, const Consts<R> *__restrict__ consts,
                                             const int *__restrict__ tsim, const R *__restrict__ state,
                                             int *__restrict__ pos) {
  __shared__ int s_best[NT / 32];
  const int t = blockIdx.x, s = __ldg(tsim + t);
  if (!consts[s].shift) return;
  const SimDesc sd = sims[s];
  const int lt = t - sd.tile0, by = lt / sd.tiles_x, bx = lt - by * sd.tiles_x;
  const int x = by * TX + threadIdx.x / TY, y = bx * TY + threadIdx.x % TY;
  int best = 0;
  if (x < sd.g.mx && y >= 1 && y < sd.g.my) {
    const R *pl = state + sd.off_state + (long long)(N - 1) * sd.g.plane + (long long)x * sd.g.pitch;
    const R a = pl[y - 1], b = pl[y];
    if ((a - (R(1.0) - a) < R(0.0)) && (b - (R(1.0) - b) > R(0.0))) best = y + 3;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
  if ((threadIdx.x & 31) == 0) s_best[threadIdx.x >> 5] = best;
  __syncthreads();
  if (threadIdx.x == 0) {
    int b = 0;
#pragma unroll
    for (int w = 0; w < NT / 32; w++) b = max(b, s_best[w]);
    if (b > 0) atomicMax(pos + s, b);
  }
}

/* The state after the check into the other buffer: shifted by d rows where
 * pos > Shiftj, else copied.  A cell takes the cell d columns up (through
 * the boundary copy tables past the last interior column), or the liquid
 * fill beyond the ghost columns.  The first tile's thread 0 records the
 * shift for the temperature rows of the next step. */
template <typename R, int N, int K>
__global__ void __launch_bounds__(NT) ks_shift(const SimDesc *__restrict__ sims,
                                               const Consts<R> *__restrict__ consts, const int *__restrict__ tsim,
                                               const R *__restrict__ state, R *__restrict__ next,
                                               const int *__restrict__ pos, SimDyn *__restrict__ dyn) {
  const int t = blockIdx.x, s = __ldg(tsim + t);
  const Consts<R> &D = consts[s];
  const SimDesc sd = sims[s];
  const int lt = t - sd.tile0, by = lt / sd.tiles_x, bx = lt - by * sd.tiles_x;
  const int x = by * TX + threadIdx.x / TY, y = bx * TY + threadIdx.x % TY;
  const int p = pos[s];
  const int d = (D.shift && p > D.shiftj) ? p - D.shiftj : 0;
  if (lt == 0 && threadIdx.x == 0 && d > 0) {
    SimDyn &dd = dyn[s];
    dd.shift_T = dd.shift_off;
    dd.dlast = d;
    dd.fresh = 1;
    dd.shift_off += d;
    dd.pos = p;
  }
  if (x >= sd.g.mx || y >= sd.g.my) return;
  const R *src = state + sd.off_state;
  R *dst = next + sd.off_state;
  const long long row = (long long)x * sd.g.pitch, o = row + y;
  const int sy = y + d;
  if (d == 0) {
#pragma unroll
    for (int f = 0; f < N + K; f++) dst[f * sd.g.plane + o] = src[f * sd.g.plane + o];
  } else if (sy <= sd.g.my + 2) {
    const int yp = sy < sd.g.my ? sy : remap(sy, sd.g.my, D.bc_y[0][0], D.bc_y[0][1]);
    const int ym = sy < sd.g.my ? sy : remap(sy, sd.g.my, D.bc_y[1][0], D.bc_y[1][1]);
#pragma unroll
    for (int a = 0; a < N; a++) dst[a * sd.g.plane + o] = src[a * sd.g.plane + row + yp];
#pragma unroll
    for (int k = 0; k < K; k++) dst[(N + k) * sd.g.plane + o] = src[(N + k) * sd.g.plane + row + ym];
  } else {
#pragma unroll
    for (int a = 0; a < N; a++) dst[a * sd.g.plane + o] = a == N - 1 ? R(1.0) : R(0.0);
#pragma unroll
    for (int k = 0; k < K; k++) dst[(N + k) * sd.g.plane + o] = D.mu_fill[k];
  }
}

/* Flags of every tile of a state buffer from its phi (after an upload,
 * smoothing or gp_batch_set); a warp per tile row. */
template <typename R, int N>
__global__ void __launch_bounds__(NT) kf_flags(const SimDesc *__restrict__ sims, const int *__restrict__ tsim,
                                               const R *__restrict__ state, TileFlags *__restrict__ flags) {
  __shared__ unsigned s_w[TX];
  const int t = blockIdx.x;
  const SimDesc sd = sims[__ldg(tsim + t)];
  const int lt = t - sd.tile0, by = lt / sd.tiles_x, bx = lt - by * sd.tiles_x;
  const int w = threadIdx.x / TY, lane = threadIdx.x - w * TY, x = by * TX + w, y = bx * TY + lane;
  const bool valid = x < sd.g.mx && y < sd.g.my;
  int oh = -1;
  if (valid) {
    R ph[N];
#pragma unroll
    for (int a = 0; a < N; a++) ph[a] = __ldg(state + sd.off_state + a * sd.g.plane + (long long)x * sd.g.pitch + y);
    oh = one_hot<R, N>(ph);
  }
  const unsigned b = row_flag_bits<N>(valid, oh);
  if (lane == 0) s_w[w] = b;
  __syncthreads();
  if (threadIdx.x == 0) flags[t] = flags_of_rows(s_w);
}

}  // namespace gpd
