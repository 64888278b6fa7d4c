// Pair-tile kernel of uneven batches, inverse transforms (pair_tile_impl.cuh).
#include "pair_tile_impl.cuh"

namespace sipfft {

const void *pair_batch_fn_inv() { return reinterpret_cast<const void *>(pair_batch_kernel<false>); }

}  // namespace sipfft
