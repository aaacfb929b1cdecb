// D2Q9 instantiations of the fused sweep (see sweep.cuh).
#include "sweep.cuh"

namespace cflbm {

cudaError_t launch_sweep_q9(int store, int compute, const SweepArgs &a, cudaStream_t s) {
  if (compute != COMPUTE_F32) {
    switch (store) {
      case STORE_F64: return launch_sweep_t<9, double, double, 4>(a, s);
      case STORE_F32: return launch_sweep_t<9, float, double, 4>(a, s);
      case STORE_F16: return launch_sweep_t<9, F16Dev, double, 4>(a, s);
    }
  } else {
    switch (store) {
      case STORE_F64: return launch_sweep_t<9, double, float, 4>(a, s);
      case STORE_F32: return launch_sweep_t<9, float, float, 4>(a, s);
      case STORE_F16: return launch_sweep_t<9, F16Dev, float, 4>(a, s);
    }
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_sweep_channel_q9(int store, int compute, const SweepArgs &a,
                                     cudaStream_t s) {
  if (compute != COMPUTE_F32) {
    // Block fixed point: 1132x168, 400 steps 3.32 / 3.22 ms at 7 / 8 blocks per
    // SM; 400x100 1.78 / 1.79.
    switch (store) {
      case STORE_F64: return launch_sweep_channel_t<9, double, double, 8>(a, s);
      case STORE_F32: return launch_sweep_channel_t<9, float, double, 4>(a, s);
      case STORE_F16: return launch_sweep_channel_t<9, F16Dev, double, 4>(a, s);
    }
  } else {
    switch (store) {
      case STORE_F64: return launch_sweep_channel_t<9, double, float, 8>(a, s);
      case STORE_F32: return launch_sweep_channel_t<9, float, float, 8>(a, s);
      case STORE_F16: return launch_sweep_channel_t<9, F16Dev, float, 8>(a, s);
    }
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_macros_channel_q9(int store, int compute, const SweepArgs &a,
                                      cudaStream_t s) {
  if (compute != COMPUTE_F32) {
    switch (store) {
      case STORE_F64: return launch_macros_channel_t<9, double, double>(a, s);
      case STORE_F32: return launch_macros_channel_t<9, float, double>(a, s);
      case STORE_F16: return launch_macros_channel_t<9, F16Dev, double>(a, s);
    }
  } else {
    switch (store) {
      case STORE_F64: return launch_macros_channel_t<9, double, float>(a, s);
      case STORE_F32: return launch_macros_channel_t<9, float, float>(a, s);
      case STORE_F16: return launch_macros_channel_t<9, F16Dev, float>(a, s);
    }
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_stream_state_q9(int store, const SweepArgs &a, bool ref, double *out,
                                    cudaStream_t s) {
  switch (store) {
    case STORE_F64: return launch_stream_state_t<9, double>(a, ref, out, s);
    case STORE_F32: return launch_stream_state_t<9, float>(a, ref, out, s);
    case STORE_F16: return launch_stream_state_t<9, F16Dev>(a, ref, out, s);
  }
  return cudaErrorInvalidValue;
}

}  // namespace cflbm
