// Host side of the pair-tile kernels (pair_tile_impl.cuh).
#include <vector>

#include "pair_tile.cuh"
#include "sipfft_internal.h"

namespace sipfft {

// instantiated in pair_tile_fwd.cu / pair_tile_inv.cu and pair_batch_fwd.cu / pair_batch_inv.cu
const void *pair_tile_fn_fwd();
const void *pair_tile_fn_inv();
const void *pair_batch_fn_fwd();
const void *pair_batch_fn_inv();

const void *pair_kernel_fn(bool forward) { return forward ? pair_tile_fn_fwd() : pair_tile_fn_inv(); }
const void *pair_batch_fn(bool forward) { return forward ? pair_batch_fn_fwd() : pair_batch_fn_inv(); }

void pair_kernel_fns(std::vector<const void *> &out)
{
    for (int f = 0; f < 2; f++) {
        out.push_back(pair_kernel_fn(f != 0));
        out.push_back(pair_batch_fn(f != 0));
    }
    out.push_back(pair_blue_fn());
}

size_t pair_smem_bytes(int buf_words)
{
    const size_t head = ((kPairSlots * ((sizeof(PairSeg) + 15) / 16)) + 7) / 8 * 8;
    return (head + size_t(2) * buf_words) * 16;
}

cudaError_t launch_pair(const PairDesc &d, bool forward, int grid, cudaStream_t st)
{
    const size_t smem = pair_smem_bytes(d.buf_words);
    if (grid <= 0 || d.tiles == 0 || smem > static_cast<size_t>(kMaxSmemBytes)) return cudaErrorInvalidConfiguration;
    PairSeg g{};
    g.d = d;
    void *args[] = {&g};
    return launch_pdl(pair_kernel_fn(forward), dim3(grid), dim3(kPairThreads), smem, st, args);
}

cudaError_t launch_pair_blue(const PairBlue &q, int grid, cudaStream_t st)
{
    const size_t smem = pair_smem_bytes(q.g.d.buf_words);
    if (grid <= 0 || q.g.d.tiles == 0 || smem > static_cast<size_t>(kMaxSmemBytes)) return cudaErrorInvalidConfiguration;
    PairBlue g = q;
    void *args[] = {&g};
    return launch_pdl(pair_blue_fn(), dim3(grid), dim3(kPairThreads), smem, st, args);
}

cudaError_t launch_pair_batch(int grid, int buf_words, const PairSeg *segs, const int2 *items, int nitems,
                              int *words, const BatchBufs &bufs, int *err, uint32_t polls, bool forward, cudaStream_t st)
{
    BatchBufs b = bufs;
    void *args[] = {&segs, &items, &nitems, &words, &b, &err, &buf_words, &polls};
    return cudaLaunchKernel(pair_batch_fn(forward), dim3(grid), dim3(kPairThreads), args, pair_smem_bytes(buf_words), st);
}

}  // namespace sipfft
