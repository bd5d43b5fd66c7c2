// The tensor-core decode attention (sl_attn_mma.cuh) without an index list. A module of its own: with these forms beside the
// others in one module (and the row copy beside the decode kernels of sl_hash.cu) the 32-layer decode step at 32K keys took
// 807 us instead of 801 although the kernels it runs compile to the same registers: where their code lies on the device differs.
#include "sl_attn_mma.cuh"

namespace sl {

int launch_attn_dense(const AttnArgs& a, int G, cudaStream_t s) { return launch_by_shape<false, true>(a, G, s); }

}  // namespace sl
