// Descriptor of the runtime-radix kernels that transform two rows or two
// adjacent columns per thread (pair_tile.cu), and the host arithmetic that
// fills it.  Plain data and host code only: a CPU test walks the index
// arithmetic for every shape it can take.
#pragma once
#include "fft_tile.cuh"

namespace sipfft {

constexpr int kPairThreads = 128;   // threads per CTA
constexpr int kPairSlots = 3;       // descriptors in shared memory
constexpr int kPairKnown = 2048;    // producers of an uneven batch that a CTA remembers as finished
constexpr int kPairStages = 8;      // most stages of a tile
constexpr int kPairMaxRadix = 16;   // radices 2..16
constexpr int kPairBufBytes = 37504;  // most shared memory of one tile buffer (two per CTA, three CTAs per SM)
constexpr int kPairBufBytes4 = 27264;  // the same for four CTAs per SM
// Most columns (rows) of a step: a tile of 2 x 128 past the last column still has
// indices below 2^31, as FastDiv needs them (the last tile's threads look the pass
// twiddles of columns up that do not exist).
constexpr int64_t kPairMaxCols = (int64_t(1) << 31) - 2 * kPairThreads;

// Butterflies of radix R that a thread holds between a stage's gather and its
// scatter: at most 16 points of two transforms (64 registers).
constexpr int pair_nb(int R) { return 16 / R; }

struct PairStage {
    int R, ns, nbf;   // radix, product of the earlier radices, butterflies n / R of one transform
    int tasks;        // butterflies of the tile's pairs
    uint32_t ns_m;    // ceil(2^32 / ns), 0 when ns == 1
    uint32_t nbf_m;   // ceil(2^32 / nbf), 0 when nbf == 1
    int gstep;        // words between a butterfly's inputs in the work tile
    int gpad, spad;   // the boundary this stage reads / writes is padded
    int toff;         // offset of the stage's twiddle table
};

// The work tile holds one 16-byte word (re 0, re 1, im 0, im 1) per element of
// each of its P pairs, element e of pair p at word p * SP + e * SE.  Rows are
// stored one after the other (SE = 1) and walked with the elements fastest,
// columns side by side (SP = 1) and walked with the pairs fastest.
struct PairDesc {
    const void *in;
    void *out;
    int n, io, nstages;
    int P, lp;        // pairs per tile (columns: a power of two and its log2)
    int SE, SP;
    int descending;   // last tile first (single steps)
    int rows;         // 1: contiguous rows, 0: columns
    int runs;         // last stage walked with the elements fastest (columns stored contiguously)
    int buf_words;    // 16-byte words of one tile buffer
    PairStage st[kPairStages];
    int64_t n_cols, n_outer;
    uint32_t tiles;
    FastDiv dv_tiles, dv_block, dv_gdiv, dv_gns, dv_post;
    Addr in_a, out_a;  // rows: row distances in in_a.dist / out_a.dist
    // 32-bit copies of the strides that the stages use, and the distance of the
    // odd column of a pair from the even one (-1: crosses column blocks, computed)
    uint32_t in_es, out_es, out_cs;
    int32_t out_jump, out_delta;
    const float2 *stw;  // per-stage twiddle tables
    const float2 *tw;   // exp(-2 pi i k / 2n) of the packed real kinds
    int g_twiddle;
    const float2 *g_t1, *g_t2, *g_lo, *g_hi;
    int g_log2l;
    int64_t g_step;
};

// One segment of an uneven batch on the pair kernel (offsets in bytes into
// the buffers of BatchBufs; dep: the segment whose output this one reads and
// its tile count; consumed: another segment reads this one's output).
struct alignas(16) PairSeg {
    PairDesc d;
    int64_t in_off, out_off;
    int in_buf, out_buf;
    int dep, dep_tiles, consumed;
};

// A Bluestein transform in one kernel (pair_blue_kernel): rows of length nb as a
// circular convolution of length d.n, both FFTs in shared memory.
struct alignas(16) PairBlue {
    PairSeg g;  // g.d: rows of d.n points; in / out as for the other kernels
    const float2 *chirp, *bmul;
    int64_t in_dist, out_dist;  // float2 (real sides: float) elements between rows
    int nb, kind;               // TileDesc::blue_n, blue_kind
};

// Relative cost per point of a tile of P pairs: every thread runs every
// butterfly slot of a stage (about eight instructions of addressing,
// shared-memory and twiddle work per point and the butterfly's FP32 operations,
// halved by packing; about 24 per butterfly for its indices), a tile costs about
// 350 instructions a thread besides, and columns in row runs below 128 bytes
// waste memory transactions.
inline double pair_tile_cost(int n, const int *radix, int nstages, bool rows, int P, int buf_words)
{
    static const double flops[] = {0, 0, 2, 5.3, 4, 7.2, 7.3, 11, 6.5, 11.5, 9.2, 18, 9.3, 22, 13, 12.5, 9.3};
    double c = 350.0;
    for (int s = 0; s < nstages; s++) c += pair_nb(radix[s]) * (24.0 + radix[s] * (8.0 + flops[radix[s]]));
    c *= double(kPairThreads) / (double(n) * P);
    if (buf_words * 16 > kPairBufBytes4) c *= 1.12;
    if (!rows) c *= P >= 8 ? 1.0 : (P == 4 ? 1.15 : (P == 2 ? 1.6 : 2.5));
    return c;
}

// Tile shape for a transform of length n with these radices and P pairs per
// tile (columns: a power of two): every stage must fit the threads' butterflies
// and the staged rows (raw_dist elements apart; columns: n) a tile buffer.
inline bool pair_shape(PairDesc &d, int n, const int *radix, int nstages, bool rows, bool runs, int64_t raw_dist, int P,
                       int max_buf = kPairBufBytes)
{
    if (n < 2 || nstages < 1 || nstages > kPairStages || P < 1 || P > kPairThreads) return false;
    d.n = n;
    d.nstages = nstages;
    d.rows = rows ? 1 : 0;
    d.runs = runs ? 1 : 0;
    int lp = 0;
    while ((1 << lp) < P) lp++;
    if ((1 << lp) != P && !rows) return false;
    for (int s = 0; s < nstages; s++)
        if (radix[s] < 2 || radix[s] > kPairMaxRadix || int64_t(n / radix[s]) * P > kPairThreads * pair_nb(radix[s]))
            return false;
    // rows: an odd R0 scatters without conflicts; columns: eight pairs fill the banks
    const bool padded = nstages > 1 && radix[0] % 2 == 0 && (rows || P < 8);
    d.P = P;
    d.lp = lp;
    d.SE = rows ? 1 : (runs ? P | 1 : P);
    const int elems = n + (padded ? n / radix[0] : 0);
    d.SP = rows ? elems | 1 : 1;
    const int64_t work = rows ? int64_t(P - 1) * d.SP + elems : int64_t(elems - 1) * d.SE + P;
    const int64_t raw = rows ? (2 * P * raw_dist + 3) / 2 : int64_t(n) * P;
    const int64_t words = ((work > raw ? work : raw) + 7) / 8 * 8;
    if (words * 16 > max_buf) return false;
    d.buf_words = static_cast<int>(words);
    int ns = 1, toff = 0;
    for (int s = 0; s < nstages; s++) {
        PairStage &t = d.st[s];
        t.R = radix[s];
        t.ns = ns;
        t.nbf = n / radix[s];
        t.tasks = t.nbf * P;
        t.ns_m = ns_reciprocal(ns);
        t.nbf_m = ns_reciprocal(t.nbf);
        t.gpad = padded && s == 1;
        t.spad = padded && s == 0;
        t.gstep = (t.nbf + (t.gpad ? t.nbf / radix[0] : 0)) * d.SE;
        t.toff = toff;
        if (s > 0) toff += (radix[s] - 1) * ns;
        ns *= radix[s];
    }
    return ns == n;
}

// Butterfly b of thread tid in a stage of `tasks` butterflies, nbf of each transform: pair p,
// index j; off (and butterfly 0) beyond the tile.  E: the elements fastest, else the pairs.
struct PairTask {
    int p, j;
    bool on;
};
template <bool E>
__host__ __device__ __forceinline__ PairTask pair_task(int tid, int b, int lp, int nbf, uint32_t nbf_m, int tasks)
{
    if constexpr (E) {
        const int i = tid + b * kPairThreads;
        const bool on = i < tasks;
        const int u = on ? i : 0;
#ifdef __CUDA_ARCH__
        const int p = nbf == 1 ? u : static_cast<int>(__umulhi(static_cast<uint32_t>(u), nbf_m));
#else
        const int p = nbf == 1 ? u : static_cast<int>((uint64_t(uint32_t(u)) * nbf_m) >> 32);
#endif
        return {p, u - p * nbf, on};
    } else {
        const int j = (tid >> lp) + b * (kPairThreads >> lp);
        const bool on = j < nbf;
        return {tid & ((1 << lp) - 1), on ? j : 0, on};
    }
}

// Work-tile words of butterfly (p, j) of stage t: its first input (the others
// follow t.gstep apart) and its first output (ns * SE apart).
__host__ __device__ __forceinline__ int pair_gather_at(int SP, int SE, int gpad, int p, int j, int q)
{
    return p * SP + (j + (gpad ? q : 0)) * SE;  // q = j div ns
}
__host__ __device__ __forceinline__ int pair_scatter_at(int SP, int SE, int spad, int ns, int R, int p, int j, int q)
{
    return p * SP + (j + q * ns * (R - 1) + (spad ? j : 0)) * SE;  // q ns R + (j - q ns)
}

}  // namespace sipfft
