// Device code of the runtime-radix tiles of two transforms per thread: columns of a strided axis
// or of a pass of a long transform, contiguous rows (C2C, and even-length R2C /
// C2R through the packed half), and the uneven batch's segments.
//
// The one-transform runtime engine (stages.cuh, fft_tile.cu) spends about 170
// instructions per point and pass: padded shared-memory indices, stage and
// pass twiddles and the element copies are computed for every point.  Here a
// thread owns the same butterfly of two adjacent rows or columns: one 16-byte
// shared-memory word, one address and one twiddle serve both, the butterflies
// run as packed FP32 instructions, the work tile's layout is affine in the
// butterfly's input and output index (no per-element padding arithmetic), and
// the tile is copied in 16-byte pieces.  Radices up to 16 are compiled, so
// most lengths up to 256 take two stages.
//
// A CTA has 128 threads and two tile buffers of 20 to 37 KB: the next tile's
// copies (cp.async) are in flight while this one is transformed in place.
// Four CTAs fit an SM (three with tiles above 27 KB), with 128 registers a
// thread; the data of a stage (up to 16 points of two transforms) stays in
// registers across the barrier between its gather and its scatter.
#pragma once
#include "async_copy.cuh"
#include "pair_engine.cuh"
#include "pair_tile.cuh"
#include "sipfft_internal.h"

namespace sipfft {

namespace {

__device__ __forceinline__ void cp_async16(void *dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// ------------------------------------------------------------------------------------ tile copies
// Rows: the tile is one run of elements; it lands one element in when its
// first element is not 16-byte aligned, so that the rest copies in 16-byte
// pieces.  Columns: [element][P pairs], 16 bytes a pair where aligned.
__device__ __forceinline__ int64_t pair_row_start(const PairDesc &d, uint32_t t) { return int64_t(t) * (2 * d.P) * d.in_a.dist; }

__device__ __forceinline__ void pair_issue(const PairDesc &d, const void *in, float4 *buf, uint32_t t)
{
    const int tid = threadIdx.x;
    const float2 *x = static_cast<const float2 *>(in);
    if (d.rows) {
        const int64_t left = d.n_cols - int64_t(t) * (2 * d.P);
        const int rows = left < 2 * d.P ? static_cast<int>(left) : 2 * d.P;
        const int own = d.io == IO_C2R_PACKED ? d.n + 1 : d.n;  // elements of a row (the distance may be larger)
        const int count = static_cast<int>((rows - 1) * d.in_a.dist) + own;
        const float2 *src = x + pair_row_start(d, t);
        const int mis = (reinterpret_cast<uintptr_t>(src) >> 3) & 1;
        float2 *dst = reinterpret_cast<float2 *>(buf) + mis;
        if (mis && tid == 0) cp_async8(dst, src);
        const int chunks = (count - mis) >> 1;
#pragma unroll 4
        for (int i = tid; i < chunks; i += kPairThreads) cp_async16(dst + mis + 2 * i, src + mis + 2 * i);
        if (((count - mis) & 1) && tid == 0) cp_async8(dst + count - 1, src + count - 1);
        return;
    }
    const uint32_t o = d.dv_tiles.div(t);
    const int p = tid & (d.P - 1);
    const int64_t c = int64_t(t - o * d.dv_tiles.d) * (2 * d.P) + 2 * p;
    if (c >= d.n_cols) return;
    const uint32_t es = d.in_es;
    const float2 *src = x + o * d.in_a.dist + c + static_cast<uint64_t>(static_cast<uint32_t>(tid) >> d.lp) * es;
    float4 *dst = buf + tid;
    const uint64_t step = static_cast<uint64_t>(kPairThreads >> d.lp) * es;
    const int total = d.n * d.P;
    if (c + 1 < d.n_cols) {
        if (((reinterpret_cast<uintptr_t>(src) & 15) == 0) && es % 2 == 0) {
#pragma unroll 4
            for (int i = tid; i < total; i += kPairThreads, dst += kPairThreads, src += step) cp_async16(dst, src);
        } else {
#pragma unroll 4
            for (int i = tid; i < total; i += kPairThreads, dst += kPairThreads, src += step) {
                cp_async8(dst, src);
                cp_async8(reinterpret_cast<float2 *>(dst) + 1, src + 1);
            }
        }
    } else {
        for (int i = tid; i < total; i += kPairThreads, dst += kPairThreads, src += step) cp_async8(dst, src);
    }
}

// ------------------------------------------------------------------------------------ stages
// A CTA's shared memory: slots for the segments (descriptors) of the tile
// being transformed and of the next two, then the two tile buffers.
constexpr int kPairSlotWords = (sizeof(PairSeg) + 15) / 16;
constexpr int kPairHeadWords = (kPairSlots * kPairSlotWords + 7) / 8 * 8;

extern __shared__ __align__(128) float4 pair_smem[];

__device__ __forceinline__ PairSeg &pair_slot(int slot)
{
    return *reinterpret_cast<PairSeg *>(pair_smem + slot * kPairSlotWords);
}

// What the stages of one tile need besides the descriptor.
struct PairTileState {
    int slot;           // descriptor
    int buf;            // first word of the tile buffer
    int mis;            // rows: elements that the staged rows start into the buffer
    float2 *out;        // outputs of the tile's outer index
    uint32_t c0;        // first column (rows: first row) of the tile
    uint32_t left;      // columns (rows) from c0 on
};

__device__ __forceinline__ cpx2 word_in(float4 q) { return {make_float2(q.x, q.y), make_float2(q.z, q.w)}; }
__device__ __forceinline__ float4 word_of(cpx2 v) { return make_float4(v.re.x, v.re.y, v.im.x, v.im.y); }

// Where a stage reads, and how the threads walk the tile: rows with the
// elements fastest, columns with the pairs fastest; a work tile either way (the
// last stage of columns whose outputs are contiguous takes the elements fastest).
// (Twiddled columns of the longest rows, whose t1 is not built, have stages of their own: the
// lookup's registers slowed the others by up to 12 %, 96000 x 43 40 -> 45 us.)
enum PairSource {
    kPairRows = 0, kPairCols = 1, kPairColsTwiddled = 2, kPairColsTwiddled2 = 3, kPairWorkE = 4, kPairWorkP = 5
};

// One stage of radix R: reads the staged tile (rows, columns, columns with the
// inter-pass twiddles of a multi-pass step) or the work tile, writes the work
// tile or (to_global) the outputs.  A function of its own: nothing lives in
// registers across stages.  Threads beyond the tile's butterflies run butterfly
// 0 again and store nothing, so that no load hangs on a branch.
template <int R, PairSource SRC, bool FWD>
__device__ __noinline__ void pair_stage(int stage, bool to_global, const PairTileState s)
{
    constexpr int NB = pair_nb(R);
    constexpr bool TWIDDLED = SRC == kPairColsTwiddled || SRC == kPairColsTwiddled2;
    constexpr bool FIRST = SRC <= kPairColsTwiddled2;
    constexpr bool E = SRC == kPairRows || SRC == kPairWorkE;  // elements fastest
    const PairDesc &d = pair_slot(s.slot).d;
    const PairStage &t = d.st[stage];
    const int tid = static_cast<int>(threadIdx.x);
    // (copied out of shared memory once: stores and barriers would reload them)
    const int nbf = t.nbf, ns = FIRST ? 1 : t.ns, lp = d.lp, tasks = t.tasks, SP = d.SP, SE = d.SE, spad = t.spad;
    const uint32_t ns_m = t.ns_m, nbf_m = t.nbf_m;
    cpx2 v[NB * R];
    const int p0 = tid & ((1 << lp) - 1);
    auto task = [&](int b, int &p, int &j) -> bool {
        const PairTask k = pair_task<E>(tid, b, lp, nbf, nbf_m, tasks);
        p = k.p;
        j = k.j;
        return k.on;
    };
    auto block = [&](int j) { return FIRST ? j : static_cast<int>(__umulhi(static_cast<uint32_t>(j), ns_m)); };  // j div ns
    PassTwiddle tw{};
    PassTable2 two{};
    if constexpr (TWIDDLED) {
        const uint32_t c = s.c0 + 2 * p0;
        tw = PassTwiddle{d.g_t1, d.g_t2, d.dv_gns.d, d.dv_gns.mod(d.dv_gdiv.div(c)), d.dv_gns.mod(d.dv_gdiv.div(c + 1))};
        if constexpr (SRC == kPairColsTwiddled2)
            two = PassTable2{d.g_lo, d.g_hi, d.g_log2l, static_cast<uint32_t>(d.g_step)};
    }
#pragma unroll
    for (int b = 0; b < NB; b++) {
        int p, j;
        task(b, p, j);
        if constexpr (SRC == kPairRows) {
            const int dist = static_cast<int>(d.in_a.dist);
            const float2 *x0 = reinterpret_cast<const float2 *>(pair_smem + s.buf) + s.mis + (2 * p) * dist + j;
            const float2 *x1 = static_cast<uint32_t>(2 * p + 1) < s.left ? x0 + dist : x0;
#pragma unroll
            for (int r = 0; r < R; r++) v[b * R + r] = pair_of(x0[r * nbf], x1[r * nbf]);
        } else if constexpr (FIRST) {
            const float4 *w = pair_smem + s.buf + (j << lp) + p;
            const int step = nbf << lp;
#pragma unroll
            for (int r = 0; r < R; r++) {
                const float4 u = w[r * step];
                v[b * R + r] = pair_of(make_float2(u.x, u.y), make_float2(u.z, u.w));
            }
            if constexpr (SRC == kPairColsTwiddled)
                tw.template apply<R, FWD, false>(v + b * R, tw.at<false>(tw.t1, j));
            if constexpr (SRC == kPairColsTwiddled2)
                tw.template apply<R, FWD, false>(v + b * R, pair_of(two.at(j, tw.k0), two.at(j, tw.k1)));
        } else {
            const int q = block(j);
            const float4 *w = pair_smem + s.buf + pair_gather_at(SP, SE, t.gpad, p, j, q);
            const int step = t.gstep;
#pragma unroll
            for (int r = 0; r < R; r++) v[b * R + r] = word_in(w[r * step]);
            const float2 *wt = d.stw + t.toff + (j - q * ns);
#pragma unroll
            for (int r = 1; r < R; r++) v[b * R + r] = cmul(v[b * R + r], dir<FWD>(__ldg(wt + (r - 1) * ns)));
        }
        dft<R, FWD>(v + b * R);
    }
    if (to_global) {
        const uint32_t es = d.out_es;
        const uint64_t step = static_cast<uint64_t>(static_cast<uint32_t>(ns)) * es;
        const int delta0 = d.out_delta, jump = d.out_jump;
        const uint32_t cs = d.out_cs;
        const FastDiv by_block = d.dv_block;
        // first element of the even column of pair p, and the odd column's distance
        auto column = [&](int p, int64_t &delta) -> float2 * {
            const uint32_t c = s.c0 + 2 * p;
            const uint32_t blk = jump ? by_block.div(c) : 0u;
            delta = delta0 >= 0 ? delta0 : int64_t(cs) + int64_t(by_block.div(c + 1) - blk) * jump;
            return s.out + (static_cast<uint64_t>(c) * cs + static_cast<uint64_t>(blk) * static_cast<uint32_t>(jump));
        };
        int64_t delta = 0;
        float2 *base = E ? nullptr : column(p0, delta);
#pragma unroll
        for (int b = 0; b < NB; b++) {
            int p, j;
            if (task(b, p, j) && static_cast<uint32_t>(2 * p) < s.left) {
                if constexpr (E) base = column(p, delta);
                float2 *y0 = base + static_cast<uint64_t>(static_cast<uint32_t>(j)) * es;
                const bool second = static_cast<uint32_t>(2 * p + 1) < s.left;
                if (!E && second && delta == 1 && ((reinterpret_cast<uintptr_t>(y0) & 15) == 0) && es % 2 == 0) {
#pragma unroll
                    for (int r = 0; r < R; r++, y0 += step) st_stream(y0, first_of(v[b * R + r]), second_of(v[b * R + r]));
                } else {
                    float2 *y1 = y0 + delta;
#pragma unroll
                    for (int r = 0; r < R; r++, y0 += step) st_stream(y0, first_of(v[b * R + r]));
                    if (second) {
#pragma unroll
                        for (int r = 0; r < R; r++, y1 += step) st_stream(y1, second_of(v[b * R + r]));
                    }
                }
            }
        }
        return;
    }
    __syncthreads();
#pragma unroll
    for (int b = 0; b < NB; b++) {
        int p, j;
        if (task(b, p, j)) {
            float4 *w = pair_smem + s.buf + pair_scatter_at(SP, SE, spad, ns, R, p, j, block(j));
            const int step = ns * SE;
#pragma unroll
            for (int r = 0; r < R; r++) w[r * step] = word_of(v[b * R + r]);
        }
    }
    __syncthreads();
}

#define SIPFFT_PAIR_RADICES(X) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15) X(16)

template <PairSource SRC, bool FWD>
__device__ __forceinline__ void pair_any(int R, int stage, bool to_global, const PairTileState &s)
{
#define SIPFFT_PAIR(RR) \
    case RR: pair_stage<RR, SRC, FWD>(stage, to_global, s); break;
    switch (R) {
        SIPFFT_PAIR_RADICES(SIPFFT_PAIR)
        default: break;  // the planner only emits the radices above
    }
#undef SIPFFT_PAIR
}

// The real kinds' passes over the pairs of bins k and m-k of every row hold
// kRealUnroll pairs in flight per thread.
constexpr int kRealUnroll = 4;

// R2C post-twiddle of the packed transforms in the work tile: bins k and m-k
// of every row (r2c_pair on two rows at once).
template <bool FWD>
__device__ __noinline__ void pair_r2c_post(const PairTileState s)
{
    const PairDesc &d = pair_slot(s.slot).d;
    const int m = d.n, half = m / 2 + 1, SP = d.SP;
    const int64_t dist = d.out_a.dist;
    const FastDiv by_half = d.dv_post;
    const float2 *tw = d.tw;
    // (the pairs of rows that exist)
    const uint32_t total = static_cast<uint32_t>(half) * min(static_cast<uint32_t>(d.P), (s.left + 1) / 2);
    for (uint32_t i0 = threadIdx.x; i0 < total; i0 += kRealUnroll * kPairThreads) {
        cpx2 zk[kRealUnroll], zm[kRealUnroll];
        float2 w[kRealUnroll];
#pragma unroll
        for (int u = 0; u < kRealUnroll; u++) {
            const uint32_t i = min(i0 + u * kPairThreads, total - 1);
            const int p = static_cast<int>(by_half.div(i)), k = static_cast<int>(i) - p * half;
            const float4 *z = pair_smem + s.buf + p * SP;
            zk[u] = word_in(z[k]);
            zm[u] = word_in(z[k == 0 ? 0 : m - k]);
            w[u] = __ldg(tw + k);
        }
#pragma unroll
        for (int u = 0; u < kRealUnroll; u++) {
            const uint32_t i = i0 + u * kPairThreads;
            if (i < total) {
                const int p = static_cast<int>(by_half.div(i)), k = static_cast<int>(i) - p * half;
                // X[k] = S/2 + w U/2, X[m-k] = conj(S/2 - w U/2), S = Z[k] + conj Z[m-k], U = -i (Z[k] - conj Z[m-k])
                const cpx2 S = cscale(cadd(zk[u], cconj(zm[u])), 0.5f);
                const cpx2 D = cscale(csub(zk[u], cconj(zm[u])), 0.5f);
                const cpx2 wu = cmul(cneg(mul_i(D)), dir<FWD>(w[u]));
                const cpx2 a = cadd(S, wu), b = cconj(csub(S, wu));
                float2 *y = s.out + (s.c0 + 2 * p) * dist + k;
                const bool second = static_cast<uint32_t>(2 * p + 1) < s.left, both_bins = 2 * k != m;
                st_stream(y, first_of(a));
                if (both_bins) st_stream(y + (m - 2 * k), first_of(b));
                if (second) {
                    y += dist;
                    st_stream(y, second_of(a));
                    if (both_bins) st_stream(y + (m - 2 * k), second_of(b));
                }
            }
        }
    }
}

// C2R pre-twiddle of the staged half spectra in place: Z[k] and Z[m-k] of the
// packed m-point sequence take the places of X[k] and X[m-k] (see C2RPre).
template <bool FWD>
__device__ __noinline__ void pair_c2r_pre(const PairTileState s)
{
    const PairDesc &d = pair_slot(s.slot).d;
    const int m = d.n, half = m / 2 + 1, dist = static_cast<int>(d.in_a.dist);
    const FastDiv by_half = d.dv_post;
    const float2 *tw = d.tw;
    const uint32_t total = static_cast<uint32_t>(half) * min(static_cast<uint32_t>(d.P), (s.left + 1) / 2);
    float2 *raw = reinterpret_cast<float2 *>(pair_smem + s.buf) + s.mis;
    for (uint32_t i0 = threadIdx.x; i0 < total; i0 += kRealUnroll * kPairThreads) {
        cpx2 xk[kRealUnroll], xm[kRealUnroll];
        float2 w[kRealUnroll];
        // a pair of bins is read and written by one thread only; the clamped rounds
        // beyond `total` read the last pair and write nothing
#pragma unroll
        for (int u = 0; u < kRealUnroll; u++) {
            const uint32_t i = min(i0 + u * kPairThreads, total - 1);
            const int p = static_cast<int>(by_half.div(i)), k = static_cast<int>(i) - p * half;
            const float2 *x0 = raw + (2 * p) * dist, *x1 = static_cast<uint32_t>(2 * p + 1) < s.left ? x0 + dist : x0;
            xk[u] = pair_of(x0[k], x1[k]);
            xm[u] = pair_of(x0[m - k], x1[m - k]);
            w[u] = __ldg(tw + k);
        }
#pragma unroll
        for (int u = 0; u < kRealUnroll; u++) {
            const uint32_t i = i0 + u * kPairThreads;
            if (i < total) {
                const int p = static_cast<int>(by_half.div(i)), k = static_cast<int>(i) - p * half;
                float2 *x0 = raw + (2 * p) * dist, *x1 = static_cast<uint32_t>(2 * p + 1) < s.left ? x0 + dist : x0;
                if (k == 0) xk[u].im = xm[u].im = make_float2(0.f, 0.f);
                const cpx2 ev = cadd(xk[u], cconj(xm[u]));
                const cpx2 od = cmul(csub(xk[u], cconj(xm[u])), dir<FWD>(w[u]));
                const cpx2 zk = cadd_i(ev, od), zm = cconj(csub_i(ev, od));
                x0[k] = first_of(zk);
                x1[k] = second_of(zk);
                if (k != 0 && 2 * k != m) {
                    x0[m - k] = first_of(zm);
                    x1[m - k] = second_of(zm);
                }
            }
        }
    }
}

// Stages of one staged tile (a barrier after its copies is the caller's).
// REAL: the descriptor may be a packed real kind (not in the uneven batch).
template <bool FWD, bool REAL>
__device__ __forceinline__ void pair_tile(int slot, int buf, const void *in, void *out, uint32_t t)
{
    const PairDesc &d = pair_slot(slot).d;
    PairTileState s;
    s.slot = slot;
    s.buf = buf;
    s.mis = 0;
    if (d.rows) {
        s.out = static_cast<float2 *>(out);
        s.mis = static_cast<int>((reinterpret_cast<uintptr_t>(static_cast<const float2 *>(in) + pair_row_start(d, t)) >> 3) & 1);
        s.c0 = t * (2 * d.P);
    } else {
        const uint32_t o = d.dv_tiles.div(t);
        s.c0 = (t - o * d.dv_tiles.d) * (2 * d.P);
        s.out = static_cast<float2 *>(out) + int64_t(o) * d.out_a.dist;
    }
    s.left = static_cast<uint32_t>(d.n_cols) - s.c0;
    const int S = d.nstages, io = d.io;
    const bool direct = !REAL || io != IO_R2C_PACKED;  // R2C: the post-twiddle writes the outputs
    if constexpr (REAL) {
        if (io == IO_C2R_PACKED) {
            pair_c2r_pre<FWD>(s);
            __syncthreads();
        }
    }
    if (d.rows)
        pair_any<kPairRows, FWD>(d.st[0].R, 0, S == 1 && direct, s);
    else if (d.g_twiddle && d.g_t1)
        pair_any<kPairColsTwiddled, FWD>(d.st[0].R, 0, S == 1, s);
    else if (d.g_twiddle)
        pair_any<kPairColsTwiddled2, FWD>(d.st[0].R, 0, S == 1, s);
    else
        pair_any<kPairCols, FWD>(d.st[0].R, 0, S == 1, s);
#pragma unroll 1
    for (int i = 1; i < S; i++) {
        const bool last = i == S - 1;
        if (d.rows || (last && d.runs))
            pair_any<kPairWorkE, FWD>(d.st[i].R, i, last && direct, s);
        else
            pair_any<kPairWorkP, FWD>(d.st[i].R, i, last, s);
    }
    if constexpr (REAL) {
        if (!direct) pair_r2c_post<FWD>(s);
    }
}

__device__ __forceinline__ void copy_seg(int slot, const PairSeg *src)
{
    static_assert(sizeof(PairSeg) % 16 == 0, "segment copied as 8-byte words, slots 16-byte aligned");
    const uint64_t *s = reinterpret_cast<const uint64_t *>(src);
    uint64_t *d = reinterpret_cast<uint64_t *>(&pair_slot(slot));
    for (int i = threadIdx.x; i < static_cast<int>(sizeof(PairSeg) / 8); i += kPairThreads) d[i] = s[i];
}

template <bool FWD>
__global__ void __launch_bounds__(kPairThreads, 4) pair_tile_kernel(const __grid_constant__ PairSeg g)
{
    copy_seg(0, &g);
    pdl_wait();
    __syncthreads();
    const PairDesc &d = pair_slot(0).d;
    const uint32_t tiles = g.d.tiles;
    const int words = g.d.buf_words;
    auto at = [&](uint32_t t) { return g.d.descending ? tiles - 1 - t : t; };
    uint32_t t = blockIdx.x;
    if (t < tiles) pair_issue(d, g.d.in, pair_smem + kPairHeadWords, at(t));
    for (int i = 0; t < tiles; t += gridDim.x, i++) {
        const uint32_t tn = t + gridDim.x;
        cp_async_wait_all();
        __syncthreads();  // this tile has landed, and the previous one's buffer is free
        if (tn < tiles)
            pair_issue(d, g.d.in, pair_smem + kPairHeadWords + ((i + 1) & 1) * words, at(tn));
        else
            pdl_launch_dependents();
        pair_tile<FWD, true>(0, kPairHeadWords + (i & 1) * words, g.d.in, g.d.out, at(t));
    }
}

// ------------------------------------------------------------------------------------ Bluestein
// y[k] = chirp[k] IFFT_M(FFT_M(x chirp) bmul)[k] of two rows per thread: one read
// of x, one write of y, both FFTs in shared memory (as two launches the M-point
// intermediate went through HBM and the tiles ran on the one-transform kernel:
// 1021 x 4096 204 us).  The inverse FFT is conj(FFT(conj .)).  Two tile buffers:
// the first FFT works in one, the product is staged as rows in the other.
template <int KIND>
__device__ __forceinline__ float2 blue_in(const void *in, int64_t base, int e, int nb)
{
    if constexpr (KIND == 1) {
        return make_float2(static_cast<const float *>(in)[base + e], 0.f);
    } else if constexpr (KIND == 2) {
        const float2 *x = static_cast<const float2 *>(in) + base;
        if (2 * e > nb) return cconj(x[nb - e]);
        float2 v = x[e];
        if (e == 0 || 2 * e == nb) v.y = 0.f;
        return v;
    } else {
        return static_cast<const float2 *>(in)[base + e];
    }
}

// The element-wise passes hold kBlueUnroll elements' loads in flight per thread (one
// at a time the loads' latency was half of the kernel: 122 us at 1021 x 4096).
constexpr int kBlueUnroll = 8;

template <int KIND>
__device__ __forceinline__ void blue_load(const PairBlue &q, int m, int rows, int64_t row0, float2 *raw)
{
    const int nb = q.nb;
    for (int e0 = threadIdx.x; e0 < m; e0 += kBlueUnroll * kPairThreads) {
        float2 c[kBlueUnroll];
#pragma unroll
        for (int u = 0; u < kBlueUnroll; u++) {
            const int e = e0 + u * kPairThreads;
            c[u] = e < nb ? __ldg(q.chirp + e) : make_float2(0.f, 0.f);
        }
        for (int l = 0; l < rows; l++) {
            float2 x[kBlueUnroll];
#pragma unroll
            for (int u = 0; u < kBlueUnroll; u++) {
                const int e = e0 + u * kPairThreads;
                x[u] = e < nb ? blue_in<KIND>(q.g.d.in, (row0 + l) * q.in_dist, e, nb) : make_float2(0.f, 0.f);
            }
#pragma unroll
            for (int u = 0; u < kBlueUnroll; u++) {
                const int e = e0 + u * kPairThreads;
                if (e < m) raw[l * m + e] = e < nb ? cmul(x[u], c[u]) : make_float2(0.f, 0.f);
            }
        }
    }
}

__device__ __forceinline__ void pair_row_stages(const PairTileState &s)
{
    const PairDesc &d = pair_slot(s.slot).d;
    pair_any<kPairRows, true>(d.st[0].R, 0, false, s);
#pragma unroll 1
    for (int i = 1; i < d.nstages; i++) pair_any<kPairWorkE, true>(d.st[i].R, i, false, s);
}

__global__ void __launch_bounds__(kPairThreads, 4) pair_blue_kernel(const __grid_constant__ PairBlue q)
{
    copy_seg(0, &q.g);
    pdl_wait();
    __syncthreads();
    const int m = q.g.d.n, P = q.g.d.P, SP = q.g.d.SP, words = q.g.d.buf_words;
    float4 *A = pair_smem + kPairHeadWords, *B = A + words;
    for (uint32_t t = blockIdx.x; t < q.g.d.tiles; t += gridDim.x) {
        const int64_t row0 = int64_t(t) * (2 * P);
        const int rows = static_cast<int>(min(int64_t(2 * P), q.g.d.n_cols - row0)), pairs = (rows + 1) / 2;
        float2 *raw = reinterpret_cast<float2 *>(A);
        if (q.kind == 0)
            blue_load<0>(q, m, rows, row0, raw);
        else if (q.kind == 1)
            blue_load<1>(q, m, rows, row0, raw);
        else
            blue_load<2>(q, m, rows, row0, raw);
        if (t + gridDim.x >= q.g.d.tiles) pdl_launch_dependents();
        __syncthreads();
        PairTileState s{0, kPairHeadWords, 0, nullptr, 0u, static_cast<uint32_t>(rows)};
        pair_row_stages(s);
        raw = reinterpret_cast<float2 *>(B);
        for (int e0 = threadIdx.x; e0 < m; e0 += kBlueUnroll * kPairThreads) {
            float2 c[kBlueUnroll];
#pragma unroll
            for (int u = 0; u < kBlueUnroll; u++) {
                const int e = e0 + u * kPairThreads;
                c[u] = e < m ? __ldg(q.bmul + e) : make_float2(0.f, 0.f);
            }
            for (int p = 0; p < pairs; p++) {
#pragma unroll
                for (int u = 0; u < kBlueUnroll; u++) {
                    const int e = e0 + u * kPairThreads;
                    if (e < m) {
                        const cpx2 v = cconj(cmul(word_in(A[p * SP + e]), c[u]));
                        raw[2 * p * m + e] = first_of(v);
                        if (2 * p + 1 < rows) raw[(2 * p + 1) * m + e] = second_of(v);
                    }
                }
            }
        }
        __syncthreads();
        s.buf = kPairHeadWords + words;
        pair_row_stages(s);
        const int count = q.kind == 1 ? q.nb / 2 + 1 : q.nb;
        for (int e0 = threadIdx.x; e0 < count; e0 += kBlueUnroll * kPairThreads) {
            float2 c[kBlueUnroll];
#pragma unroll
            for (int u = 0; u < kBlueUnroll; u++) {
                const int e = e0 + u * kPairThreads;
                c[u] = e < count ? __ldg(q.chirp + e) : make_float2(0.f, 0.f);
            }
            for (int p = 0; p < pairs; p++) {
                const int64_t y0 = (row0 + 2 * p) * q.out_dist;
                const bool second = 2 * p + 1 < rows;
#pragma unroll
                for (int u = 0; u < kBlueUnroll; u++) {
                    const int e = e0 + u * kPairThreads;
                    if (e >= count) continue;
                    const cpx2 v = cmul(cconj(word_in(B[p * SP + e])), c[u]);
                    if (q.kind == 2) {
                        float *y = static_cast<float *>(q.g.d.out) + y0 + e;
                        y[0] = v.re.x;
                        if (second) y[q.out_dist] = v.re.y;
                    } else {
                        float2 *y = static_cast<float2 *>(q.g.d.out) + y0 + e;
                        st_stream(y, first_of(v));
                        if (second) st_stream(y + q.out_dist, second_of(v));
                    }
                }
            }
        }
    }
}

// ------------------------------------------------------------------------------------ uneven batches
// One persistent launch over the work list of (segment, tile) items.  A segment
// waits (bounded) for every tile of the segment whose output it reads; items are
// ordered so that producers come before their consumers.  A CTA takes its items
// from a counter and works them in the order of their tickets, so the waits end
// however many CTAs run at once: the first unfinished item of the list is the
// current item of a running CTA (or nobody's yet, and then no CTA waits), and
// every item that it could wait for comes before it.  (Items dealt by CTA number
// would need the whole grid resident, which other work on the GPU can prevent.)
//
// Everything an item needs is in shared memory before its turn: its ticket is
// drawn and its place in the list copied (cp.async) three items ahead, its
// descriptor two, its tile one (when its producer has finished; otherwise at its
// turn).  (With all of that at its turn, a chain of four
// dependent global loads stood between two tiles: barrier and long-scoreboard
// stalls were 5 of 12 cycles per instruction.)  The first tickets are drawn one
// at a time, a load apart, so that short lists spread over the CTAs.
// Finished producers are remembered, so a CTA polls each at most once more.
__device__ __forceinline__ int pair_done_count(const int *done, int dep)
{
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(done + dep) : "memory");
    return v;
}

// Polls of thread 0 until `tiles` tiles of segment dep are finished; false when it
// gives up, or another CTA has, and the words that say so are set.  (A function of
// its own: its registers would spill those of the stages.)
__device__ __noinline__ bool pair_wait(int *words, int dep, int tiles, uint32_t polls, int *err, int *status)
{
    for (uint32_t i = 0; i < polls; i++) {
        __nanosleep(128);
        if (pair_done_count(words + kBatchDone, dep) >= tiles) return true;
        if (i % 64 == 63 && *static_cast<volatile int *>(words + kBatchGaveUp) != 0) break;
    }
    atomicExch(words + kBatchGaveUp, 1);
    atomicExch(err, 2);
    *static_cast<volatile int *>(status) = 2;
    return false;
}

template <bool FWD>
__global__ void __launch_bounds__(kPairThreads, 4)
    pair_batch_kernel(const PairSeg *__restrict__ segs, const int2 *__restrict__ items, int nitems, int *words,
                      BatchBufs bufs, int *err, int buf_words, uint32_t polls)
{
    __shared__ __align__(8) int2 s_item[4];           // item k at [k & 3]
    __shared__ uint32_t s_known[kPairKnown / 32];     // producers seen finished
    __shared__ int s_flag;
    // segment whose tile this CTA finished last, -1 if nobody waits for it.  (In shared memory,
    // and no ticket held across a tile: the stages take every register, and the kernel's own that
    // live across them spill.  76 bytes of spills cost 12 %: 20000 transforms 2.85 -> 2.51 ms.)
    __shared__ int s_publish;
    const int tid = threadIdx.x;
    if (tid == 0) s_publish = -1;
    auto draw = [&]() -> uint32_t {
        return tid == 0 ? atomicAdd(reinterpret_cast<unsigned *>(words + kBatchTicket), 1u) : 0u;
    };
    for (int i = tid; i < kPairKnown / 32; i += kPairThreads) s_known[i] = 0u;
    auto place = [&](int k, uint32_t ticket) {  // list entry of this CTA's item k
        if (tid != 0) return;
        if (ticket < static_cast<uint32_t>(nitems))
            cp_async8(&s_item[k & 3], items + ticket);
        else
            s_item[k & 3] = make_int2(-1, 0);
    };
    auto describe = [&](int k) {  // its descriptor (the entry has landed)
        const int sg = s_item[k & 3].x;
        if (sg < 0) return;
        const char *src = reinterpret_cast<const char *>(segs + sg);
        char *dst = reinterpret_cast<char *>(&pair_slot(k % kPairSlots));
        for (int i = tid; i < static_cast<int>(sizeof(PairSeg) / 16); i += kPairThreads) cp_async16(dst + 16 * i, src + 16 * i);
    };
    auto source = [&](const PairSeg &g) { return static_cast<const char *>(bufs.p[g.in_buf]) + g.in_off; };
    // is the segment's producer finished?  uniform; with `wait`, polls until it is
    auto ready = [&](const PairSeg &g, bool wait) -> bool {
        const int dep = g.dep;
        if (dep < 0) return true;
        if (dep < kPairKnown && (s_known[dep >> 5] >> (dep & 31) & 1u)) return true;
        __syncthreads();  // every thread has read the bit that thread 0 may set
        if (tid == 0) {
            bool ok = pair_done_count(words + kBatchDone, dep) >= g.dep_tiles;
            if (wait && !ok) ok = pair_wait(words, dep, g.dep_tiles, polls, err, bufs.status);
            if (ok && dep < kPairKnown) s_known[dep >> 5] |= 1u << (dep & 31);
            s_flag = ok ? 1 : 0;
        }
        __syncthreads();
        return s_flag != 0;
    };
    auto copy_in = [&](int k) {
        const PairSeg &g = pair_slot(k % kPairSlots);
        pair_issue(g.d, source(g), pair_smem + kPairHeadWords + (k & 1) * buf_words, static_cast<uint32_t>(s_item[k & 3].y));
    };
    place(0, draw());
    cp_async_wait_all();
    __syncthreads();
    describe(0);
    place(1, draw());
    cp_async_wait_all();
    __syncthreads();
    // item 0 is the start of some segment's tiles: prefetched like the others
    bool staged = s_item[0].x >= 0 && ready(pair_slot(0), false);
    if (staged) copy_in(0);
    describe(1);
    place(2, draw());
    for (int k = 0;; k++) {
        // the ticket of item k + 3: its latency passes under the barrier and the copies' issue
        const uint32_t ticket = draw();
        cp_async_wait_all();
        __syncthreads();  // item k's copies, k+1's descriptor and k+2's entry have landed; item k-1 is done
        if (tid == 0 && s_publish >= 0) {
            __threadfence();
            atomicAdd(words + kBatchDone + s_publish, 1);
        }
        if (s_item[k & 3].x < 0) break;
        const PairSeg &g = pair_slot(k % kPairSlots);
        const bool more = s_item[(k + 1) & 3].x >= 0;
        if (more) describe(k + 2);
        if (!staged) {
            if (!ready(g, true)) break;  // the whole CTA: the results are incomplete, and reported as such
            copy_in(k);
            cp_async_wait_all();
            __syncthreads();
        }
        staged = more && ready(pair_slot((k + 1) % kPairSlots), false);
        if (staged) copy_in(k + 1);
        place(k + 3, ticket);
        if (tid == 0) s_publish = g.consumed ? s_item[k & 3].x : -1;
        pair_tile<FWD, false>(k % kPairSlots, kPairHeadWords + (k & 1) * buf_words, source(g),
                              static_cast<char *>(bufs.p[g.out_buf]) + g.out_off, static_cast<uint32_t>(s_item[k & 3].y));
    }
    cp_async_wait_all();
}

}  // namespace

}  // namespace sipfft
