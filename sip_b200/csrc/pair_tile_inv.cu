// Pair-tile kernel of single steps, inverse transforms (pair_tile_impl.cuh).
#include "pair_tile_impl.cuh"

namespace sipfft {

const void *pair_tile_fn_inv() { return reinterpret_cast<const void *>(pair_tile_kernel<false>); }

}  // namespace sipfft
