// The tensor-core decode attention (sl_attn_mma.cuh) without an index list. A module of its own: with these forms beside the
// others in one module the 32-layer decode step at 128K keys took 1110 us instead of 1102 although the kernels it runs
// compile to the same registers (where their code lies on the device differs).
#include "sl_attn_mma.cuh"

namespace sl {

int launch_attn_dense(const AttnArgs& a, int G, cudaStream_t s) { return launch_by_shape<false, true>(a, G, s); }

}  // namespace sl
