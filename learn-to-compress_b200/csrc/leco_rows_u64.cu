// leco_rows_u64.cu -- row encoder kernels for uint64_t columns (a translation unit per value type:
// the width-specialised packers compile in parallel).
#include "leco_rows_kernel.cuh"

namespace leco {

int launch_rows_u64(int codec, const EncodeArgs &a, bool ref, cudaStream_t st) {
  switch (codec) {
    case kLinear: return launch_rows_t<uint64_t, kLinear>(a, ref, st);
    case kFor: return launch_rows_t<uint64_t, kFor>(a, ref, st);
    case kDelta: return launch_rows_t<uint64_t, kDelta>(a, ref, st);
    case kPoly2: return launch_rows_t<uint64_t, kPoly2>(a, ref, st);
  }
  return 1;
}

}  // namespace leco
