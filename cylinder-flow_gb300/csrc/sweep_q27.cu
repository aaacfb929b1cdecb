// D3Q27 instantiations of the fused sweep (see sweep.cuh).
#include "sweep.cuh"

namespace cflbm {

cudaError_t launch_sweep_q27(int store, int compute, const SweepArgs &a, cudaStream_t s) {
  if (compute != COMPUTE_F32) {
    // Block fixed point (fixed.cuh).  REF3D 257x97x97, 20 steps and the fields: 4.83 /
    // 4.64 ms at 5 / 6 blocks per SM; FP64 operations at 3 per SM: 15.17 ms.
    switch (store) {
      case STORE_F64: return launch_sweep_t<27, double, double, 6>(a, s);
      case STORE_F32: return launch_sweep_t<27, float, double, 5>(a, s);
      case STORE_F16: return launch_sweep_t<27, F16Dev, double, 5>(a, s);
    }
  } else {
    switch (store) {
      case STORE_F64: return launch_sweep_t<27, double, float, 4>(a, s);
      case STORE_F32: return launch_sweep_t<27, float, float, 4>(a, s);
      case STORE_F16: return launch_sweep_t<27, F16Dev, float, 4>(a, s);
    }
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_sweep_channel_q27(int store, int compute, const SweepArgs &a,
                                      cudaStream_t s) {
  if (compute != COMPUTE_F32) {
    // Block fixed point: 512x128x128, 10 steps and the fields: 7.33 / 7.81 ms at 5 / 6
    // per SM; FP64 operations at 3 per SM: 22.78 ms.
    switch (store) {
      case STORE_F64: return launch_sweep_channel_t<27, double, double, 5>(a, s);
      case STORE_F32: return launch_sweep_channel_t<27, float, double, 5>(a, s);
      case STORE_F16: return launch_sweep_channel_t<27, F16Dev, double, 5>(a, s);
    }
  } else {
    switch (store) {
      // 512x128x128: 525.9 / 523.8 / 527.4 us per step at 6 / 7 / 8 per SM, 331x101x90
      // 197.7 / 194.5 / 195.9, 100x40x36 11.3 / 11.4 / 12.1
      case STORE_F64: return launch_sweep_channel_t<27, double, float, 7>(a, s);
      case STORE_F32: return launch_sweep_channel_t<27, float, float, 8>(a, s);
      case STORE_F16: return launch_sweep_channel_t<27, F16Dev, float, 8>(a, s);
    }
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_macros_channel_q27(int store, int compute, const SweepArgs &a,
                                      cudaStream_t s) {
  if (compute != COMPUTE_F32) {
    switch (store) {
      case STORE_F64: return launch_macros_channel_t<27, double, double>(a, s);
      case STORE_F32: return launch_macros_channel_t<27, float, double>(a, s);
      case STORE_F16: return launch_macros_channel_t<27, F16Dev, double>(a, s);
    }
  } else {
    switch (store) {
      case STORE_F64: return launch_macros_channel_t<27, double, float>(a, s);
      case STORE_F32: return launch_macros_channel_t<27, float, float>(a, s);
      case STORE_F16: return launch_macros_channel_t<27, F16Dev, float>(a, s);
    }
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_stream_state_q27(int store, const SweepArgs &a, bool ref, double *out,
                                    cudaStream_t s) {
  switch (store) {
    case STORE_F64: return launch_stream_state_t<27, double>(a, ref, out, s);
    case STORE_F32: return launch_stream_state_t<27, float>(a, ref, out, s);
    case STORE_F16: return launch_stream_state_t<27, F16Dev>(a, ref, out, s);
  }
  return cudaErrorInvalidValue;
}

}  // namespace cflbm
