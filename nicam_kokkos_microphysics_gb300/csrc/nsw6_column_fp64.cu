// The column phase, FP64 (nsw6_column.cuh).
#include "nsw6_column.cuh"

namespace nsw6 {

cudaError_t prepare_column_fp64(int optin) { return prepare_column<false, false>(optin); }
cudaError_t launch_column_fp64(const Problem& P, const Consts& C, cudaStream_t stream) {
  return run_column<false, false>(P, C, stream);
}

}  // namespace nsw6
