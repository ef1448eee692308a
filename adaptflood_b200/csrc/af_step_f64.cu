// af_step_f64.cu -- FP64 instantiation of the fused step.  Compiled with
// -fmad=false so each expression rounds as the reference's C++ does.
#include "af_resident.cuh"
#include "af_stream.cuh"

namespace af {
// Indices follow kStepVariant in af_step.cuh.
const void* step_kernel_f64(int variant, bool tma) {
  if (!tma) {  // large grids: bulk copies
    switch (variant) {
      case 1: return (const void*)&k_step<double, 1, 12, false>;
      case 2: return (const void*)&k_step<double, 1, 20, false>;
      case 3: return (const void*)&k_step<double, 4, 4, false>;
      case 4: return (const void*)&k_step<double, 2, 8, false>;
      default: return (const void*)&k_step<double, 1, 16, false>;
    }
  }
  switch (variant) {
    case 1: return (const void*)&k_step<double, 1, 12>;
    case 2: return (const void*)&k_step<double, 1, 20>;
    case 3: return (const void*)&k_step<double, 4, 4>;
    case 4: return (const void*)&k_step<double, 2, 8>;
    default: return (const void*)&k_step<double, 1, 16>;
  }
}
const void* batch_kernel_f64(int variant) {
  switch (variant) {
    case 1: return (const void*)&k_batch_step<double, 1, 12>;
    case 2: return (const void*)&k_batch_step<double, 1, 20>;
    case 3: return (const void*)&k_batch_step<double, 4, 4>;
    case 4: return (const void*)&k_batch_step<double, 2, 8>;
    default: return (const void*)&k_batch_step<double, 1, 16>;
  }
}
const void* stream_kernel_f64(bool tma) {
  return tma ? (const void*)&k_stream<double, true> : (const void*)&k_stream<double, false>;
}
const void* resident_kernel_f64() { return (const void*)&k_resident<double>; }
const void* batch_begin_f64() { return (const void*)&k_batch_begin<double>; }
const void* batch_fold_f64() { return (const void*)&k_batch_fold<double>; }
}  // namespace af
