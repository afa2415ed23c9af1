// The column phase, FP64 with the scheme switches (nsw6_column.cuh).
#include "nsw6_column.cuh"

namespace nsw6 {

cudaError_t prepare_column_fp64_switches(int optin) { return prepare_column<false, true>(optin); }
cudaError_t launch_column_fp64_switches(const Problem& P, const Consts& C, cudaStream_t stream) {
  return run_column<false, true>(P, C, stream);
}

}  // namespace nsw6
