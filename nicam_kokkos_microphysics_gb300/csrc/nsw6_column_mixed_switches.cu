// The column phase, mixed precision with the scheme switches (nsw6_column.cuh).
#include "nsw6_column.cuh"

namespace nsw6 {

cudaError_t prepare_column_mixed_switches(int optin) { return prepare_column<true, true>(optin); }
cudaError_t launch_column_mixed_switches(const Problem& P, const Consts& C, cudaStream_t stream) {
  return run_column<true, true>(P, C, stream);
}

}  // namespace nsw6
