#include "qmv_cluster.cuh"

namespace mtc {
cudaError_t launch_cluster_b4(cudaStream_t st, CluArgs &a, const clu::Shape &s, const clu::Plan &p) { return clu::launch_bits<4>(st, a, s, p); }
}  // namespace mtc
