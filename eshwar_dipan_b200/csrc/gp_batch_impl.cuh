/*
 * gp_batch_impl.cuh -- launchers of the batched kernels for one field type.
 * Instantiated by gp_kernels.cu, one translation unit per field type and
 * system size (FP64 without FMA contraction, so that it stays bit-identical to
 * the reference; the FP32 storage form with it); each gives a BatchLaunch table.
 */
#pragma once
#include <cuda_runtime.h>

#include "gp_fused.cuh"
#include "gp_smooth.cuh"

namespace gpd {

/* What one step's kernels are launched with.  mul: every simulation's spacings
 * are powers of two (x/dx == x*(1/dx)); diag: every phase's off-diagonal D, c_mu
 * and A are zero and no E is -0 (those terms are left out); tg: some simulation is
 * non-isothermal; solo: a batch of one's StepArgs (host memory), or NULL. */
struct StepLaunch {
  cudaStream_t stream;
  int grid;
  bool mul, diag, tg;
  bool ahead;                   /* the kernels may start while the one before them runs */
  const void *solo;
  const SimDesc *sims;
  const void *consts;
  const int4 *blist, *glist;
  BoxMaps maps;                 /* a batch of one: the maps of `state` */
  const TensorMapSlot *tmaps;   /* else, per simulation and state buffer, the maps MAP_MU and MAP_ALL (device) */
  int buf;                      /* the buffer `state` is */
  const void *state;
  void *next;
  TileFlags *flag_out;
  int *ctr;
  int ndone;                    /* the CTAs of this step's kernels together */
  StatBufs st;
};

struct BatchLaunch {
  /* set up the kernels a batch with these launch options takes (mul, diag, tg and
   * solo of l) and give the blocks per SM of its kf_bulk, kf_general and kf_step */
  cudaError_t (*prepare)(const StepLaunch &l, int *bulk, int *general, int *step);
  /* the bulk and interface lists of a step; flag_out: the flags of the buffer it
   * writes (copied into the bulk entries) */
  cudaError_t (*classify)(bool ahead, int ntiles, cudaStream_t s, const ClassifySim &solo, const SimDesc *sims, const void *consts, const int *tsim,
                          const TileFlags *flag_in, const TileFlags *flag_out, int4 *glist, int4 *blist, int *ctr);
  cudaError_t (*bulk)(const StepLaunch &l);
  cudaError_t (*general)(const StepLaunch &l);
  /* bulk and interface tiles in one launch (kf_step; not for a sums step) */
  cudaError_t (*step)(const StepLaunch &l);
  /* FP64: one step of one simulation on the caller's planes (state, next: phi;
   * solo, mul, st and stream of l) */
  cudaError_t (*direct)(const StepLaunch &l, const DirectArgs<double, true> &d, int nsm);
  /* the StepArgs of a batch of one (FP32: none, every batch takes the same kernels,
   * since another kernel's fused multiply-adds could round differently) */
  size_t solo_bytes;
  void (*solo_fill)(void *dst, const void *consts, const SimDesc *sd);
  cudaError_t (*flags)(int ntiles, cudaStream_t s, const SimDesc *sims, const int *tsim, const void *state,
                       TileFlags *flags);
  /* FP64: the listed tiles of a sweep (blocks: its blocks per SM when not NULL, no launch) */
  cudaError_t (*sweep)(const StepLaunch &l, int *blocks);
  /* FP32: one smoothing sweep of a simulation (tcc: its temperature rows, or NULL) */
  cudaError_t (*smooth)(cudaStream_t s, const void *consts, const void *phi, const void *mu, void *phin,
                        void *mun, Grid g, const double *tcc);
  /* moving frame: interface position into pos[s] (zeroed by the caller),
   * then the shifted (or copied) state into next */
  cudaError_t (*shift_pos)(int ntiles, cudaStream_t s, const SimDesc *sims, const void *consts, const int *tsim,
                           const void *state, int *pos);
  cudaError_t (*shift_apply)(int ntiles, cudaStream_t s, const SimDesc *sims, const void *consts, const int *tsim,
                             const void *state, void *next, const int *pos, SimDyn *dyn);
  /* the temperature rows of the coming step (non-isothermal simulations) */
  cudaError_t (*trows)(int nsims, cudaStream_t s, const SimDesc *sims, const void *consts, const int *ctr,
                       SimDyn *dyn, double *rows);
  size_t elem;
};

/* A launch that may (ahead) start while the kernel before it on the stream still runs:
 * the kernel waits by itself (pdl_begin) before it touches what that one writes. */
template <typename... P, typename... A>
cudaError_t launch_dependent(bool ahead, void (*k)(P...), int grid, int block, size_t smem, cudaStream_t s,
                             const A &...args) {
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3((unsigned)grid);
  c.blockDim = dim3((unsigned)block);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = ahead ? 1 : 0;
  c.attrs = &at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, k, static_cast<P>(args)...);
}

template <typename R, int N, int K, bool A>
struct BatchKernels {
  static constexpr size_t bulk_smem = bulk_smem_bytes<R, K>();
  static constexpr size_t item_smem = sizeof(TileSmem<R, N, K, A>);
  static constexpr size_t step_smem = item_smem > bulk_smem ? item_smem : bulk_smem;
  /* Kernel variants: MUL only where it can differ (FP32 always multiplies), DIAG
   * only where there are off-diagonal terms, SOLO in FP64 only; a non-isothermal
   * batch takes the TG kernels, which read each simulation's constants from global
   * memory.  f(kernel) is called with the one a launch takes. */
  static constexpr bool DIV = sizeof(R) == 8, SOLO = sizeof(R) == 8;
  static const StepArgs<R, true> &solo_of(const StepLaunch &l) {
    return *reinterpret_cast<const StepArgs<R, true> *>(l.solo);
  }
  static void solo_fill(void *dst, const void *consts, const SimDesc *sd) {
    StepArgs<R, true> *a = reinterpret_cast<StepArgs<R, true> *>(dst);
    a->c = *reinterpret_cast<const Consts<R> *>(consts);
    a->sd = *sd;
  }
  template <bool MUL, bool DIAG, typename F>
  static void with_step_md(const StepLaunch &l, F &&f) {
    if (l.tg) f(kf_step<R, N, K, A, MUL, true, false, false>, StepArgs<R, false>{});
    else if (SOLO && l.solo) f(kf_step<R, N, K, A, MUL, false, SOLO, DIAG>, pick_args(l));
    else f(kf_step<R, N, K, A, MUL, false, false, DIAG>, StepArgs<R, false>{});
  }
  static decltype(auto) pick_args(const StepLaunch &l) {
    if constexpr (SOLO) return (solo_of(l));
    else return StepArgs<R, false>{};
  }
  template <typename F>
  static void with_step(const StepLaunch &l, F &&f) {
    constexpr bool KD = K > 1;
    if (DIV && !l.mul) {
      if (KD && l.diag) with_step_md<!DIV, KD>(l, f);
      else with_step_md<!DIV, false>(l, f);
    } else {
      if (KD && l.diag) with_step_md<true, KD>(l, f);
      else with_step_md<true, false>(l, f);
    }
  }
  template <bool MUL, typename F>
  static void with_general_m(const StepLaunch &l, F &&f) {
    if (l.tg) f(kf_general<R, N, K, A, MUL, true, false>, StepArgs<R, false>{});
    else if (SOLO && l.solo) f(kf_general<R, N, K, A, MUL, false, SOLO>, pick_args(l));
    else f(kf_general<R, N, K, A, MUL, false, false>, StepArgs<R, false>{});
  }
  template <typename F>
  static void with_general(const StepLaunch &l, F &&f) {
    if (DIV && !l.mul) with_general_m<!DIV>(l, f);
    else with_general_m<true>(l, f);
  }
  template <bool MUL, typename F>
  static void with_bulk_m(const StepLaunch &l, bool sums, F &&f) {
    constexpr bool KD = K > 1;
    /* the sums step (last of a call) takes every term: same results */
    if (sums) f(kf_bulk<R, N, K, true, MUL, false>);
    else if (KD && l.diag) f(kf_bulk<R, N, K, false, MUL, KD>);
    else f(kf_bulk<R, N, K, false, MUL, false>);
  }
  template <typename F>
  static void with_bulk(const StepLaunch &l, bool sums, F &&f) {
    if (DIV && !l.mul) with_bulk_m<!DIV>(l, sums, f);
    else with_bulk_m<true>(l, sums, f);
  }
  static cudaError_t step(const StepLaunch &l) {
    cudaError_t e = cudaSuccess;
    with_step(l, [&](auto k, const auto &args) {
      e = launch_dependent(l.ahead, k, l.grid, NTI, step_smem, l.stream, args, l.sims, (const Consts<R> *)l.consts, l.blist,
                           l.glist, l.maps, l.tmaps, l.buf, (const R *)l.state, (R *)l.next, l.flag_out, l.ctr, l.ndone, l.st);
    });
    return e;
  }
  static cudaError_t bulk(const StepLaunch &l) {
    cudaError_t e = cudaSuccess;
    with_bulk(l, l.st.want_sums != 0, [&](auto k) {
      e = launch_dependent(l.ahead, k, l.grid, NTI, bulk_smem, l.stream, l.sims, (const Consts<R> *)l.consts, l.blist, l.maps, l.tmaps,
                           l.buf, (const R *)l.state, (R *)l.next, l.flag_out, l.ctr, l.ndone, l.st);
    });
    return e;
  }
  static cudaError_t general(const StepLaunch &l) {
    cudaError_t e = cudaSuccess;
    with_general(l, [&](auto k, const auto &args) {
      e = launch_dependent(l.ahead, k, l.grid, NTI, item_smem, l.stream, args, l.sims, (const Consts<R> *)l.consts, l.maps, l.tmaps,
                           l.buf, (const R *)l.state, (R *)l.next, l.flag_out, l.glist, l.ctr, l.ndone, l.st);
    });
    return e;
  }
  template <bool MUL>
  static cudaError_t direct_m(const StepLaunch &l, const DirectArgs<double, true> &d, int nsm) {
    auto k = kn_step<double, N, K, A, MUL>;
    /* on every call: the attribute belongs to the caller's context */
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)item_smem);
    if (e != cudaSuccess) return e;
    const int most = nsm * item_ctas<double, N, K, A>(), few = (d.ntiles + NOALLOC_TILES - 1) / NOALLOC_TILES;
    k<<<d.ntiles < most ? d.ntiles : (few > most ? few : most), NTI, item_smem, l.stream>>>(
        *reinterpret_cast<const StepArgs<double, true> *>(l.solo), d, (const double *)l.state, (double *)l.next, l.st);
    return cudaGetLastError();
  }
  static cudaError_t direct(const StepLaunch &l, const DirectArgs<double, true> &d, int nsm) {
    if constexpr (sizeof(R) == 8) return l.mul ? direct_m<true>(l, d, nsm) : direct_m<false>(l, d, nsm);
    else return cudaErrorNotSupported;
  }
  static cudaError_t prepare(const StepLaunch &l, int *bb, int *bg, int *bs) {
    cudaError_t e = cudaSuccess;
    auto set = [&](auto k, size_t smem, int *blocks) {
      if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e == cudaSuccess && blocks) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, k, NTI, smem);
    };
    with_bulk(l, false, [&](auto k) { set(k, bulk_smem, bb); });
    with_bulk(l, true, [&](auto k) { set(k, bulk_smem, nullptr); });
    with_general(l, [&](auto k, const auto &) { set(k, item_smem, bg); });
    with_step(l, [&](auto k, const auto &) { set(k, step_smem, bs); });
    return e;
  }
  static cudaError_t classify(bool ahead, int ntiles, cudaStream_t s, const ClassifySim &solo, const SimDesc *sims, const void *consts,
                              const int *tsim, const TileFlags *flag_in, const TileFlags *flag_out, int4 *glist,
                              int4 *blist, int *ctr) {
    return launch_dependent(ahead, kf_classify<R>, (ntiles + NTC - 1) / NTC, NTC, 0, s, solo, sims, (const Consts<R> *)consts,
                            tsim, ntiles, flag_in, flag_out, glist, blist, ctr);
  }
  static cudaError_t flags(int ntiles, cudaStream_t s, const SimDesc *sims, const int *tsim, const void *state,
                           TileFlags *fl) {
    kf_flags<R, N><<<ntiles, NT, 0, s>>>(sims, tsim, (const R *)state, fl);
    return cudaGetLastError();
  }
  static cudaError_t sweep(const StepLaunch &l, int *blocks) {
    if constexpr (sizeof(R) == 8) {
      if (blocks) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, ks_tiles<R, N, K, A>, NT, 0);
      return launch_dependent(l.ahead, ks_tiles<R, N, K, A>, l.grid, NT, 0, l.stream, l.sims, (const Consts<R> *)l.consts,
                              (const R *)l.state, (R *)l.next, l.flag_out, l.glist, l.st.trows, l.ctr, l.ndone);
    } else {
      return cudaErrorNotSupported;
    }
  }
  static cudaError_t smooth(cudaStream_t s, const void *consts, const void *phi, const void *mu, void *phin,
                            void *mun, Grid g, const double *tcc) {
    dim3 grid((g.my + 127) / 128, g.mx);
    k_smooth<R, N, K, A><<<grid, 128, 0, s>>>((const Consts<R> *)consts, (const R *)phi, (const R *)mu, (R *)phin,
                                              (R *)mun, g, tcc);
    return cudaGetLastError();
  }
  static cudaError_t shift_pos(int ntiles, cudaStream_t s, const SimDesc *sims, const void *consts, const int *tsim,
                               const void *state, int *pos) {
    ks_pos<R, N><<<ntiles, NT, 0, s>>>(sims, (const Consts<R> *)consts, tsim, (const R *)state, pos);
    return cudaGetLastError();
  }
  static cudaError_t shift_apply(int ntiles, cudaStream_t s, const SimDesc *sims, const void *consts,
                                 const int *tsim, const void *state, void *next, const int *pos, SimDyn *dyn) {
    ks_shift<R, N, K><<<ntiles, NT, 0, s>>>(sims, (const Consts<R> *)consts, tsim, (const R *)state, (R *)next, pos,
                                            dyn);
    return cudaGetLastError();
  }
  static cudaError_t trows(int nsims, cudaStream_t s, const SimDesc *sims, const void *consts, const int *ctr,
                           SimDyn *dyn, double *rows) {
    kt_rows<R><<<nsims, 128, 0, s>>>(sims, (const Consts<R> *)consts, ctr, dyn, rows);
    return cudaGetLastError();
  }
  static BatchLaunch table() {
    BatchLaunch t;
    t.prepare = prepare;
    t.classify = classify;
    t.bulk = bulk;
    t.step = step;
    t.direct = direct;
    t.solo_bytes = SOLO ? sizeof(StepArgs<R, true>) : 0;
    t.solo_fill = solo_fill;
    t.general = general;
    t.flags = flags;
    t.sweep = sweep;
    t.smooth = smooth;
    t.trows = trows;
    t.shift_pos = shift_pos;
    t.shift_apply = shift_apply;
    t.elem = sizeof(R);
    return t;
  }
};

}  // namespace gpd

/* The launch tables by field type and system size: gp_kernels.cu, one
 * translation unit per (type, NUMPHASES, components), so that they compile
 * side by side. */
#define GP_TABLE_NAME2(r, n, k) gp_batch_table_##r##_##n##_##k
#define GP_TABLE_NAME(r, n, k) GP_TABLE_NAME2(r, n, k)
#define GP_FOR_SIZES(X, r) X(r, 2, 1) X(r, 3, 1) X(r, 4, 1) X(r, 2, 2) X(r, 3, 2) X(r, 4, 2)
#define GP_DECLARE_TABLE(r, n, k) gpd::BatchLaunch GP_TABLE_NAME(r, n, k)(bool aniso);
GP_FOR_SIZES(GP_DECLARE_TABLE, double)
GP_FOR_SIZES(GP_DECLARE_TABLE, float)
#undef GP_DECLARE_TABLE
