// The 8-bit instances of the fragment kernel (one translation unit per width: they compile in parallel).
#include "qmv_frag.cuh"

namespace mtc {
cudaError_t launch_frag_b8(cudaStream_t st, const FragArgs &a, const frag::Shape &s, int sms) { return frag::launch_bits<8>(st, a, s, sms); }
}  // namespace mtc
