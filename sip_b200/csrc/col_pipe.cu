// TMA-pipelined persistent kernel for strided axes: the column pass of 2D /
// 3D plans, vertical 1D, and every pass of a multi-pass (long) transform.
//
// A tile is TB adjacent transforms of a strided axis, i.e. TB adjacent
// columns of an [outer][n][cols] array.  The tensor-memory-access engine
// copies it into shared memory as 3D boxes of TB columns x up to 256 rows
// (one rectangular copy per 256 rows, issued by one thread and completed on
// an mbarrier).  A thread transforms two adjacent columns at once (cpx2: a
// 16-byte word of the staged tile holds both), so that index arithmetic,
// shared-memory accesses and twiddle loads are paid once for two columns and
// the butterflies run as packed FP32 instructions; the last stage stores
// straight from registers to HBM, 16 bytes a thread where the columns are
// adjacent there as well.  The reference runs this axis as
// a transpose plus a DFT-matrix GEMM (core/fft/fftcore/fft_core_stride.cpp:36-188,
// ops/fft/c2c/fft_stride/fft_stride/kernel/fft_stride.cce) or as explicit
// Transpose steps around the row cores (core/fft/fft_api.cpp:527-697).
//
// Launch preconditions (the planner checks them, the exec path re-checks the
// pointer): source 16-byte aligned, column stride 1, element and outer
// strides multiples of 2 complex values (16 bytes), column and tile counts
// below 2^31.
#include <cuda.h>

#include "sipfft_internal.h"
#include "pair_engine.cuh"

namespace sipfft {

namespace {

// L2 policy of the tile loads.  Out of place no later step of the plan reads the
// input again while the outputs are the next step's input: the input's lines
// leave L2 first (65536 x 256 113 -> 110 us, 2^20 x 16 124 -> 121).  In place the
// same lines are written back at once and keep the normal priority (2048^2 x 8
// 209 us, 218 with evict-first loads).
__device__ __forceinline__ uint64_t load_policy(bool in_place)
{
    uint64_t first, normal;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(first));
    asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(normal));
    return in_place ? normal : first;
}

// 3D tiled bulk-tensor load of box {x: columns, y: rows, z: outer} into shared memory
__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, int x, int y, int z, uint64_t *bar,
                                            uint64_t policy)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, "
        "{%2, %3, %4}], [%5], %6;" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar)), "l"(policy)
        : "memory");
}

}  // namespace

// Shared memory of one CTA: barriers, two tile buffers, and with PP a work tile.
// COUT: contiguous column outputs (pair_last_runs).
template <class Q, int T, int P, bool PP, bool COUT>
struct ColShape {
    using Tile = PairTile<Q, P, COUT ? P + 1 : P>;
    static constexpr int kThreads = P * T;
    static constexpr int kTileWords = P * Q::N;  // 16-byte words
    static constexpr int kBufWords = PP || Tile::kWords < kTileWords ? kTileWords : Tile::kWords;
    static constexpr size_t kSmem = 128 + (size_t(2) * kBufWords + (PP ? Tile::kWords : 0)) * sizeof(float4);
    static constexpr int kPerSm = static_cast<int>(size_t(228 * 1024) / (kSmem + 1024));
    static_assert(kPerSm >= 1 && Q::N / T == 16 && kBufWords % 8 == 0, "tile shape");
};

// Two tile buffers: the next tile streams into one while the other is
// transformed.  descending: the last tile first, so that a step starts with what
// the step before it wrote last, which is still in L2 (256^3 140 -> 130 us, 256^2 x 256
// 97 -> 87, 65536 x 256 116 -> 113).  The work tile takes the staged tile's place once stage 0 has
// read it; with PP (2048 points, one CTA per SM) it has memory of its own, which
// saves the barrier in between.  Measured on 65536 x 256: a staging tile of its
// own, refilled after stage 0, left too few bytes in flight.
template <class Q, int T, int P, bool PP, bool COUT, bool FWD>
__global__ void __launch_bounds__(ColShape<Q, T, P, PP, COUT>::kThreads, ColShape<Q, T, P, PP, COUT>::kPerSm)
    col_pipe_kernel(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ TileDesc d, int *err,
                    int descending)
{
    pdl_enter();
    using Shape = ColShape<Q, T, P, PP, COUT>;
    using Tile = typename Shape::Tile;
    constexpr int N = Q::N, TB = 2 * P;
    constexpr int BOX = N < 256 ? N : 256;
    constexpr int NBOX = N / BOX;
    extern __shared__ __align__(128) unsigned char smraw[];
    uint64_t *bars = reinterpret_cast<uint64_t *>(smraw);
    float4 *bufs = reinterpret_cast<float4 *>(smraw + 128);
    const int tid = threadIdx.x;
    const int p = tid % P, lane = tid / P;
    float2 *out = static_cast<float2 *>(d.out);
    const uint32_t tiles = static_cast<uint32_t>(d.num_tiles);
    const uint32_t cols = static_cast<uint32_t>(d.n_cols);

    if (tid == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        fence_barrier_init();
    }
    __syncthreads();

    const uint64_t policy = load_policy(d.in == d.out);
    auto issue = [&](uint32_t t, int b) {
        if (tid == 0) {
            if (descending) t = tiles - 1 - t;
            const uint32_t o = d.dv_tiles.div(t), c0 = (t - o * d.dv_tiles.d) * TB;
            float4 *dst = bufs + b * Shape::kBufWords;
            fence_proxy_async_smem();
            mbar_arrive_expect_tx(&bars[b], static_cast<uint32_t>(Shape::kTileWords * sizeof(float4)));
#pragma unroll
            for (int k = 0; k < NBOX; k++)
                tma_load_3d(dst + k * BOX * P, &tmap, static_cast<int>(c0), k * BOX, static_cast<int>(o), &bars[b],
                            policy);
        }
    };

    uint32_t t = blockIdx.x;
    if (t < tiles) issue(t, 0);
    for (int i = 0; t < tiles; t += gridDim.x, i++) {
        const int b = i & 1;
        const uint32_t tn = t + gridDim.x;
        if (tn < tiles) issue(tn, b ^ 1);
        // a thread whose bounded wait gave up still runs the tile (every access
        // stays in bounds) and the CTA leaves together at the end of the iteration
        const bool timed_out = !mbar_wait_bounded(&bars[b], (i >> 1) & 1);
        if (timed_out) atomicExch(err, 1);
        const uint32_t u = descending ? tiles - 1 - t : t;
        const uint32_t o = d.dv_tiles.div(u), ct = (u - o * d.dv_tiles.d) * TB, c0 = ct + 2 * p;
        PassTwiddle tw{nullptr, nullptr, 0, 0, 0};
        if (d.g_twiddle) {
            tw.t1 = d.g_t1;
            tw.t2 = d.g_t2;
            tw.ns = d.dv_gns.d;
            tw.k0 = d.dv_gns.mod(d.dv_gdiv.div(c0));
            tw.k1 = d.dv_gns.mod(d.dv_gdiv.div(c0 + 1));
        }
        float4 *buf = bufs + b * Shape::kBufWords;
        float4 *work = PP ? bufs + 2 * Shape::kBufWords : buf;
        cpx2 v[static_maxv<Q, T>()];
        pair_stage0<Q, T, P, FWD>(v, buf + p, lane, tw,
                                  PassTable2{d.g_lo, d.g_hi, d.g_log2l, static_cast<uint32_t>(d.g_step)});
        if constexpr (!PP) __syncthreads();
        sscatter<Q, 0, T>(v, typename Tile::template Row<0>{work + p}, lane, true);
        __syncthreads();
        if constexpr (COUT) {
            pair_last_runs<Q, T, P, P + 1, FWD>(
                v, work, tid, cols - ct,
                [&](int c) { return out + col_base32(d.out_a, d.dv_block, o, ct + c); }, d.stw);
        } else {
            const int64_t b0 = col_base32(d.out_a, d.dv_block, o, c0), b1 = col_base32(d.out_a, d.dv_block, o, c0 + 1);
            const bool wide = b1 == b0 + 1 && ((reinterpret_cast<uintptr_t>(out + b0) & 15) == 0) &&
                              d.out_a.estride % 2 == 0 && c0 + 1 < cols;
            pair_stages<Q, T, P, FWD, 1>(v, work + p,
                                         PairColumns{out + b0, out + b1, d.out_a.estride, c0 + 1 < cols, wide}, lane,
                                         c0 < cols, d.stw);
        }
        // the buffers are free for the copy issued in iteration i+1; a CTA-uniform exit after a timeout
        if (__syncthreads_or(timed_out)) return;
    }
}

// ------------------------------------------------------------------------------------ host side
namespace {

struct ColPipeEntry {
    int n, tpt, tb;
    size_t smem[2];
    int nstages, radix[4];
    const void *fn[2][2];  // [contiguous column outputs][forward]
};

template <class Q, int T, int P, bool PP = false>
ColPipeEntry col_entry()
{
    ColPipeEntry e{Q::N, T, 2 * P, {ColShape<Q, T, P, PP, false>::kSmem, 0}, Q::S, {},
                   {{reinterpret_cast<const void *>(col_pipe_kernel<Q, T, P, PP, false, false>),
                     reinterpret_cast<const void *>(col_pipe_kernel<Q, T, P, PP, false, true>)},
                    {nullptr, nullptr}}};
    for (int s = 0; s < Q::S; s++) e.radix[s] = Q::r[s];
    if constexpr (P >= 8 && Q::S == 2) {
        e.smem[1] = ColShape<Q, T, P, PP, true>::kSmem;
        e.fn[1][0] = reinterpret_cast<const void *>(col_pipe_kernel<Q, T, P, PP, true, false>);
        e.fn[1][1] = reinterpret_cast<const void *>(col_pipe_kernel<Q, T, P, PP, true, true>);
    }
    return e;
}

// Engines with 16 points of two columns per thread.  Tiles of 32 KB (16 KB for
// 64 points), 64 and 128 threads: three to six CTAs per SM and up to 168
// registers a thread; 128-byte row runs up to 256 points, 64 and 32 bytes for
// 512 and 1024 points.  2048 points: 64 KB tiles, one CTA of 256 threads.
const std::vector<ColPipeEntry> &col_registry()
{
    static const std::vector<ColPipeEntry> r = {
        col_entry<Seq<16, 2>, 2, 32>(),     col_entry<Seq<16, 4>, 4, 16>(),     col_entry<Seq<16, 8>, 8, 16>(),    col_entry<Seq<16, 16>, 16, 8>(),
        col_entry<Seq<16, 16, 2>, 32, 4>(), col_entry<Seq<16, 16, 4>, 64, 2>(), col_entry<Seq<16, 16, 8>, 128, 2, true>(),
    };
    return r;
}

using EncodeTiledFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                   const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn()
{
    static EncodeTiledFn fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            return static_cast<EncodeTiledFn>(nullptr);
        }
        return reinterpret_cast<EncodeTiledFn>(p);
    }();
    return fn;
}

}  // namespace

bool col_pipe_kernel(int n, bool forward, bool contiguous_out, ColPipe &c)
{
    for (const ColPipeEntry &e : col_registry())
        if (e.n == n) {
            const int k = contiguous_out && e.fn[1][0] ? 1 : 0;
            c = ColPipe{e.fn[k][forward ? 1 : 0], e.tpt, e.tb, e.smem[k], e.nstages,
                        {e.radix[0], e.radix[1], e.radix[2], e.radix[3]}};
            return true;
        }
    return false;
}

bool col_pipe_has_engine(int n)
{
    ColPipe c;
    return col_pipe_kernel(n, true, false, c);
}

void col_pipe_kernel_fns(std::vector<const void *> &out)
{
    for (const ColPipeEntry &e : col_registry())
        for (int k = 0; k < 2; k++)
            for (int f = 0; f < 2; f++)
                if (e.fn[k][f]) out.push_back(e.fn[k][f]);
}

// At least half a tile of columns: below that the element-copy tiles waste less.
bool col_pipe_layout_ok(const TileDesc &d)
{
    const Addr &a = d.in_a;
    const int64_t most = int64_t(1) << 31;
    return 2 * d.n_cols >= d.tb && a.cstride == 1 && a.cblock == 0 && a.estride % 2 == 0 && a.estride > 0 &&
           (d.n_outer == 1 || a.dist % 2 == 0) && d.n_outer < most && d.tiles_per_outer * d.tb < most &&
           d.num_tiles < most && d.out_a.cblock < most && d.g_div < most && d.g_ns < most && encode_fn() != nullptr;
}

cudaError_t launch_col_pipe(const void *fn, const TileDesc &d, size_t smem, int grid, bool descending, int *err,
                            cudaStream_t st)
{
    if (!fn || grid <= 0 || (reinterpret_cast<uintptr_t>(d.in) & 15)) return cudaErrorInvalidConfiguration;
    EncodeTiledFn enc = encode_fn();
    if (!enc) return cudaErrorNotSupported;
    const int n = d.n;
    const int box_rows = n < 256 ? n : 256;
    CUtensorMap map;
    // complex64 elements moved as opaque 8-byte words
    const cuuint64_t dims[3] = {static_cast<cuuint64_t>(d.n_cols), static_cast<cuuint64_t>(n),
                                static_cast<cuuint64_t>(d.n_outer)};
    const int64_t outer_stride = d.n_outer > 1 ? d.in_a.dist : d.in_a.estride * n + (d.in_a.estride * n) % 2;
    const cuuint64_t strides[2] = {static_cast<cuuint64_t>(d.in_a.estride) * 8,
                                   static_cast<cuuint64_t>(outer_stride) * 8};
    const cuuint32_t box[3] = {static_cast<cuuint32_t>(d.tb), static_cast<cuuint32_t>(box_rows), 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = enc(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, const_cast<void *>(d.in), dims, strides, box,
                           estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return cudaErrorInvalidValue;
    TileDesc dd = d;
    int down = descending ? 1 : 0;
    void *args[] = {&map, &dd, &err, &down};
    return launch_pdl(fn, dim3(grid), dim3(d.tb / 2 * d.tpt), smem, st, args);
}

}  // namespace sipfft
