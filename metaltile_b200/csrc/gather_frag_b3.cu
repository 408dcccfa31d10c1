#include "gather_frag.cuh"

namespace mtc {
cudaError_t launch_gather_frag_b3(cudaStream_t st, const GfArgs &a, const gfrag::Shape &s, const gfrag::Plan &p, int sms) { return gfrag::launch_bits<3>(st, a, s, p, sms); }
}  // namespace mtc
