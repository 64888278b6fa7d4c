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
        for (int i = tid; i < chunks; i += kPairThreads) cp_async16(dst + mis + 2 * i, src + mis + 2 * i);
        if (((count - mis) & 1) && tid == 0) cp_async8(dst + count - 1, src + count - 1);
        return;
    }
    const uint32_t o = d.dv_tiles.div(t);
    const int p = tid & (d.P - 1);
    const int64_t c = int64_t(t - o * d.dv_tiles.d) * (2 * d.P) + 2 * p;
    if (c >= d.n_cols) return;
    const int64_t es = d.in_a.estride;
    const float2 *src = x + o * d.in_a.dist + c + (tid >> d.lp) * es;
    float4 *dst = buf + tid;
    const int64_t step = (kPairThreads >> d.lp) * es;
    const int total = d.n * d.P;
    if (c + 1 < d.n_cols) {
        if (((reinterpret_cast<uintptr_t>(src) & 15) == 0) && es % 2 == 0) {
            for (int i = tid; i < total; i += kPairThreads, dst += kPairThreads, src += step) cp_async16(dst, src);
        } else {
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
// A CTA's shared memory: two slots for the segments (descriptors) of the tile
// being transformed and of the next one, then the two tile buffers.
constexpr int kPairSlotWords = (sizeof(PairSeg) + 15) / 16;
constexpr int kPairHeadWords = (2 * kPairSlotWords + 7) / 8 * 8;

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
    float2 *out;
    uint32_t o, c0;     // outer index and first column (rows: first row) of the tile
    uint32_t left;      // columns (rows) from c0 on
};

__device__ __forceinline__ cpx2 word_in(float4 q) { return {make_float2(q.x, q.y), make_float2(q.z, q.w)}; }
__device__ __forceinline__ float4 word_of(cpx2 v) { return make_float4(v.re.x, v.re.y, v.im.x, v.im.y); }

enum PairSource { kPairWork = 0, kPairRows = 1, kPairCols = 2, kPairColsTwiddled = 3 };

// One stage of radix R: reads the staged tile (rows, columns, columns with the
// inter-pass twiddles of a multi-pass step) or the work tile, writes the work
// tile or (to_global) the outputs.  A function of its own: nothing lives in
// registers across stages.  Threads beyond the tile's butterflies run butterfly
// 0 again and store nothing, so that no load hangs on a branch.
template <int R, PairSource SRC, bool FWD>
__device__ __noinline__ void pair_stage(int stage, bool to_global, const PairTileState s)
{
    constexpr int NB = pair_nb(R);
    constexpr bool FIRST = SRC != kPairWork;
    const PairDesc &d = pair_slot(s.slot).d;
    const PairStage &t = d.st[stage];
    const int nbf = t.nbf, tasks = t.tasks, ns = FIRST ? 1 : t.ns, lp = d.lp;
    const bool fast_e = SRC == kPairRows || d.rows || (to_global && d.runs);  // elements fastest
    const uint32_t nbf_m = t.nbf_m, ns_m = t.ns_m;
    cpx2 v[NB * R];
    // butterfly b of this thread: pair p, index j, block q = j div ns
    auto task = [&](int b, int &p, int &j, int &q) {
        int i = static_cast<int>(threadIdx.x) + b * kPairThreads;
        const bool on = i < tasks;
        i = on ? i : 0;
        if (fast_e) {
            p = nbf == 1 ? i : static_cast<int>(__umulhi(static_cast<uint32_t>(i), nbf_m));
            j = i - p * nbf;
        } else {
            p = i & ((1 << lp) - 1);
            j = i >> lp;
        }
        q = FIRST ? j : static_cast<int>(__umulhi(static_cast<uint32_t>(j), ns_m));
        return on;
    };
#pragma unroll
    for (int b = 0; b < NB; b++) {
        int p, j, q;
        task(b, p, j, q);
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
            if constexpr (SRC == kPairColsTwiddled) {
                const uint32_t c = s.c0 + 2 * p;
                const PassTwiddle tw{d.g_t1, d.g_t2, d.dv_gns.d, d.dv_gns.mod(d.dv_gdiv.div(c)),
                                     d.dv_gns.mod(d.dv_gdiv.div(c + 1))};
                const PassTable2 two{d.g_lo, d.g_hi, d.g_log2l, static_cast<uint32_t>(d.g_step)};
                tw.template apply<R, FWD, false>(v + b * R, j, two);
            }
        } else {
            const float4 *w = pair_smem + s.buf + pair_gather_at(d, t, p, j, q);
            const int step = t.gstep;
#pragma unroll
            for (int r = 0; r < R; r++) v[b * R + r] = word_in(w[r * step]);
            const float2 *tw = d.stw + t.toff + (j - q * ns);
#pragma unroll
            for (int r = 1; r < R; r++) v[b * R + r] = cmul(v[b * R + r], dir<FWD>(__ldg(tw + (r - 1) * ns)));
        }
        dft<R, FWD>(v + b * R);
    }
    if (to_global) {
        const int64_t es = d.out_a.estride, step = ns * es;
#pragma unroll
        for (int b = 0; b < NB; b++) {
            int p, j, q;
            if (task(b, p, j, q) && static_cast<uint32_t>(2 * p) < s.left) {
                const uint32_t c = s.c0 + 2 * p;
                const bool second = static_cast<uint32_t>(2 * p + 1) < s.left;
                float2 *y0 = s.out + col_base32(d.out_a, d.dv_block, s.o, c) + j * es;
                float2 *y1 = s.out + col_base32(d.out_a, d.dv_block, s.o, c + 1) + j * es;
                if (second && y1 == y0 + 1 && ((reinterpret_cast<uintptr_t>(y0) & 15) == 0) && es % 2 == 0) {
#pragma unroll
                    for (int r = 0; r < R; r++, y0 += step) st_stream(y0, first_of(v[b * R + r]), second_of(v[b * R + r]));
                } else {
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
        int p, j, q;
        if (task(b, p, j, q)) {
            float4 *w = pair_smem + s.buf + pair_scatter_at(d, t, p, j, q);
            const int step = ns * d.SE;
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

// R2C post-twiddle of the packed transforms in the work tile: bins k and m-k
// of every row (r2c_pair on two rows at once).
template <bool FWD>
__device__ __noinline__ void pair_r2c_post(const PairTileState s)
{
    const PairDesc &d = pair_slot(s.slot).d;
    const int m = d.n, half = m / 2 + 1;
    const int64_t dist = d.out_a.dist;
    const uint32_t total = static_cast<uint32_t>(half * d.P);
    for (uint32_t i = threadIdx.x; i < total; i += kPairThreads) {
        const int p = static_cast<int>(d.dv_post.div(i)), k = static_cast<int>(i) - p * half;
        if (static_cast<uint32_t>(2 * p) >= s.left) break;
        const float4 *w = pair_smem + s.buf + p * d.SP;
        const cpx2 zk = word_in(w[k]), zm = word_in(w[k == 0 ? 0 : m - k]);
        // X[k] = S/2 + w U/2, X[m-k] = conj(S/2 - w U/2), S = Z[k] + conj Z[m-k], U = -i (Z[k] - conj Z[m-k])
        const cpx2 S = cscale(cadd(zk, cconj(zm)), 0.5f);
        const cpx2 D = cscale(csub(zk, cconj(zm)), 0.5f);
        const cpx2 wu = cmul(cneg(mul_i(D)), dir<FWD>(__ldg(d.tw + k)));
        const cpx2 a = cadd(S, wu), b = cconj(csub(S, wu));
        float2 *y = s.out + (s.c0 + 2 * p) * dist;
        const bool second = static_cast<uint32_t>(2 * p + 1) < s.left;
        st_stream(y + k, first_of(a));
        if (second) st_stream(y + dist + k, second_of(a));
        if (2 * k != m) {
            st_stream(y + m - k, first_of(b));
            if (second) st_stream(y + dist + m - k, second_of(b));
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
    const uint32_t total = static_cast<uint32_t>(half * d.P);
    for (uint32_t i = threadIdx.x; i < total; i += kPairThreads) {
        const int p = static_cast<int>(d.dv_post.div(i)), k = static_cast<int>(i) - p * half;
        if (static_cast<uint32_t>(2 * p) >= s.left) break;
        float2 *x0 = reinterpret_cast<float2 *>(pair_smem + s.buf) + s.mis + (2 * p) * dist;
        float2 *x1 = static_cast<uint32_t>(2 * p + 1) < s.left ? x0 + dist : x0;
        cpx2 xk = pair_of(x0[k], x1[k]), xm = pair_of(x0[m - k], x1[m - k]);
        if (k == 0) xk.im = xm.im = make_float2(0.f, 0.f);
        const cpx2 ev = cadd(xk, cconj(xm));
        const cpx2 od = cmul(csub(xk, cconj(xm)), dir<FWD>(__ldg(d.tw + k)));
        const cpx2 zk = cadd_i(ev, od), zm = cconj(csub_i(ev, od));
        x0[k] = first_of(zk);
        x1[k] = second_of(zk);
        if (k != 0 && 2 * k != m) {
            x0[m - k] = first_of(zm);
            x1[m - k] = second_of(zm);
        }
    }
}

// Stages of one staged tile (a barrier after its copies is the caller's).
template <bool FWD>
__device__ __forceinline__ void pair_tile(int slot, int buf, const void *in, void *out, uint32_t t)
{
    const PairDesc &d = pair_slot(slot).d;
    PairTileState s;
    s.slot = slot;
    s.buf = buf;
    s.out = static_cast<float2 *>(out);
    s.mis = 0;
    if (d.rows) {
        s.mis = static_cast<int>((reinterpret_cast<uintptr_t>(static_cast<const float2 *>(in) + pair_row_start(d, t)) >> 3) & 1);
        s.o = 0;
        s.c0 = t * (2 * d.P);
    } else {
        s.o = d.dv_tiles.div(t);
        s.c0 = (t - s.o * d.dv_tiles.d) * (2 * d.P);
    }
    s.left = static_cast<uint32_t>(d.n_cols) - s.c0;
    const int S = d.nstages, io = d.io;
    const bool direct = io != IO_R2C_PACKED;  // R2C: the post-twiddle writes the outputs
    if (io == IO_C2R_PACKED) {
        pair_c2r_pre<FWD>(s);
        __syncthreads();
    }
    if (d.rows)
        pair_any<kPairRows, FWD>(d.st[0].R, 0, S == 1 && direct, s);
    else if (d.g_twiddle)
        pair_any<kPairColsTwiddled, FWD>(d.st[0].R, 0, S == 1, s);
    else
        pair_any<kPairCols, FWD>(d.st[0].R, 0, S == 1, s);
#pragma unroll 1
    for (int i = 1; i < S; i++) pair_any<kPairWork, FWD>(d.st[i].R, i, i == S - 1 && direct, s);
    if (!direct) pair_r2c_post<FWD>(s);
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
    uint32_t t = blockIdx.x;
    if (t < tiles) pair_issue(d, g.d.in, pair_smem + kPairHeadWords, t);
    cp_async_commit();
    for (int i = 0; t < tiles; t += gridDim.x, i++) {
        const uint32_t tn = t + gridDim.x;
        // the other buffer was released by the barrier that ended the previous tile
        if (tn < tiles)
            pair_issue(d, g.d.in, pair_smem + kPairHeadWords + ((i + 1) & 1) * words, tn);
        else
            pdl_launch_dependents();
        cp_async_commit();
        cp_async_wait<1>();
        __syncthreads();
        pair_tile<FWD>(0, kPairHeadWords + (i & 1) * words, g.d.in, g.d.out, t);
        __syncthreads();
    }
    cp_async_wait<0>();
}

// ------------------------------------------------------------------------------------ uneven batches
// The work list of batch_fft_kernel (fft_tile.cu) on pair tiles: items
// (segment, tile) are dequeued in order from a global counter, a segment waits
// (bounded) for every tile of the segment whose output it reads, and the CTA's
// next item is dequeued and, when its producer has finished, copied in while
// the current one computes.  Items are ordered so that producers are dequeued
// before their consumers and every CTA is resident, so the waits end.
__device__ __forceinline__ bool pair_dep_done(const PairSeg *segs, int *done, int dep)
{
    if (dep < 0) return true;
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(done + dep) : "memory");
    return v >= static_cast<int>(segs[dep].d.tiles);
}
__device__ __forceinline__ bool pair_dep_wait(const PairSeg *segs, int *done, int dep, int *err)
{
    for (uint32_t poll = 0; poll < (1u << 24); poll++) {
        if (pair_dep_done(segs, done, dep)) return true;
        __nanosleep(128);
    }
    atomicExch(err, 2);
    return false;
}
template <bool FWD>
__global__ void __launch_bounds__(kPairThreads, 4)
    pair_batch_kernel(const PairSeg *__restrict__ segs, const int2 *__restrict__ items, int nitems, int *counter,
                      int *done, BatchBufs bufs, int *err, int buf_words)
{
    // [i & 1]: the item computed in iteration i (the next item's slots are
    // written while the current item's are still read)
    __shared__ int2 s_item[2];
    __shared__ int s_ok, s_pref[2];
    const int tid = threadIdx.x;
    auto dequeue = [&](int slot) {
        const int w = atomicAdd(counter, 1);
        int2 it = make_int2(-1, 0);
        int ready = 0;
        if (w < nitems) {
            it = items[w];
            ready = pair_dep_done(segs, done, segs[it.x].dep);
        }
        s_item[slot] = it;
        s_pref[slot] = ready;
    };
    auto source = [&](const PairSeg &g) { return static_cast<const char *>(bufs.p[g.in_buf]) + g.in_off; };
    // copies slot's segment and, when its producer has finished, starts its tile
    auto fetch = [&](int slot) {
        if (s_item[slot].x >= 0) {
            copy_seg(slot, segs + s_item[slot].x);
            __syncthreads();
            const PairSeg &g = pair_slot(slot);
            if (s_pref[slot])
                pair_issue(g.d, source(g), pair_smem + kPairHeadWords + slot * buf_words, static_cast<uint32_t>(s_item[slot].y));
        }
        cp_async_commit();
    };
    if (tid == 0) dequeue(0);
    __syncthreads();
    fetch(0);
    for (int i = 0; s_item[i & 1].x >= 0; i++) {
        const int cur = i & 1, nx = cur ^ 1, buf = kPairHeadWords + cur * buf_words;
        // the previous iteration's item, whose slots and buffer these are, ended with a barrier
        if (tid == 0) dequeue(nx);
        __syncthreads();
        fetch(nx);
        const PairSeg &g = pair_slot(cur);
        const int2 it = s_item[cur];
        bool ok = true;
        if (!s_pref[cur]) {
            if (tid == 0) s_ok = pair_dep_wait(segs, done, g.dep, err) ? 1 : 0;
            __syncthreads();
            ok = s_ok != 0;
            if (ok) pair_issue(g.d, source(g), pair_smem + buf, static_cast<uint32_t>(it.y));
            cp_async_commit();
            cp_async_wait<0>();
        } else {
            cp_async_wait<1>();  // the current item's copies have landed
        }
        __syncthreads();
        if (ok) pair_tile<FWD>(cur, buf, source(g), static_cast<char *>(bufs.p[g.out_buf]) + g.out_off, static_cast<uint32_t>(it.y));
        __syncthreads();
        if (ok && tid == 0) {
            __threadfence();
            atomicAdd(done + it.x, 1);
        }
    }
    cp_async_wait<0>();
}

}  // namespace

}  // namespace sipfft
