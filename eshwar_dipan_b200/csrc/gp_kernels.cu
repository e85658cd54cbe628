/*
 * gp_kernels.cu -- the step and smoothing kernels of one field type GP_R and
 * one system size (GP_N phases, GP_K components), compiled once per
 * combination: GP_R=double without FMA contraction (bit-identical to the
 * reference), GP_R=float, the FP32 storage form, with it.
 */
#include "gp_batch_impl.cuh"

gpd::BatchLaunch GP_TABLE_NAME(GP_R, GP_N, GP_K)(bool aniso) {
  return aniso ? gpd::BatchKernels<GP_R, GP_N, GP_K, true>::table()
               : gpd::BatchKernels<GP_R, GP_N, GP_K, false>::table();
}
