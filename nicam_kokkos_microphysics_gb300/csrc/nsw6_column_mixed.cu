// The column phase, mixed precision (nsw6_column.cuh).
#include "nsw6_column.cuh"

namespace nsw6 {

cudaError_t prepare_column_mixed(int optin) { return prepare_column<true, false>(optin); }
cudaError_t launch_column_mixed(const Problem& P, const Consts& C, cudaStream_t stream) {
  return run_column<true, false>(P, C, stream);
}

}  // namespace nsw6
