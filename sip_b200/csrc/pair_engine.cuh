// Compile-time FFT stages on two transforms per thread (cpx2), shared by the
// column kernels: the work tile in shared memory, the staged input with the
// inter-pass twiddles of a multi-pass step, and the stores of the last stage.
//
// Why two: the one-transform engines are bound by instruction issue at about
// 60 % FP32 arithmetic.  With two transforms a thread the arithmetic issues as
// packed instructions and everything else (addresses, shared-memory and
// twiddle loads, barriers) is paid once for both.
#pragma once
#include "static_engine.cuh"

namespace sipfft {

// Work tile of P pairs: the 16-byte word (re 0, re 1, im 0, im 1) of element e
// of pair p at e * P + p, so that eight threads of adjacent pairs (or, for
// P < 8, of adjacent elements) touch eight adjacent words.  With P < 8 and an
// even first radix the scatter of stage 0, whose threads write R0 elements
// apart, would hit the same banks: its boundary skips P words every R0 elements.
// With PITCH = P + 1 words an element (P = 8 and more), threads of adjacent
// elements hit different banks as well: the last stage can then be read with
// the elements fastest (pair_last_runs).
template <class Q, int P, int PITCH = P>
struct PairTile {
    static constexpr int R0 = Q::r[0];
    static constexpr bool kPad = P < 8 && R0 % 2 == 0;
    static constexpr int kWords = PITCH * (Q::N + (kPad ? Q::N / R0 : 0));
    template <int B>
    struct Row {
        float4 *w;  // tile + p
        __device__ __forceinline__ static int at(int e)
        {
            return (e + (B == 0 && kPad ? static_cast<int>(static_cast<unsigned>(e) / R0) : 0)) * PITCH;
        }
        __device__ __forceinline__ cpx2 operator()(int e) const
        {
            const float4 q = w[at(e)];
            return {make_float2(q.x, q.y), make_float2(q.z, q.w)};
        }
        __device__ __forceinline__ void operator()(int e, cpx2 v) const
        {
            w[at(e)] = make_float4(v.re.x, v.re.y, v.im.x, v.im.y);
        }
    };
};

// Stage 0 of a pair of adjacent columns from the staged tile (interleaved
// complex values, [element][P pairs]).  A multi-pass step multiplies element
// e = j + r N/R0 of Stockham column k by W^(e k) = t1[j][k] t2[r][k]: both
// tables are contiguous in k, adjacent columns read adjacent entries, and the
// product of two rounded entries is as exact as the two-level table lookup (rms
// 3.3e-8 either way).  Against that lookup (two gathers at computed indices for
// every element of every column) it needs no index arithmetic per element.
// Where t1 is not built (more than 8 MB) its entries come from two short tables
// of roots less one (root_product: 2.1e-8; a third rounded factor would make the
// product 4.0e-8).
struct PassTable2 {
    const float2 *lo, *hi;  // exp(-2 pi i m / F) - 1, m < 2^log2l, and for multiples of 2^log2l
    int log2l;
    uint32_t step;
    __device__ __forceinline__ float2 at(int e, uint32_t k) const
    {
        const uint32_t m = static_cast<uint32_t>(e) * k * step;
        return root_product(__ldg(lo + (m & ((1u << log2l) - 1u))), __ldg(hi + (m >> log2l)));
    }
};

struct PassTwiddle {
    const float2 *t1, *t2;  // rows of `ns` entries; nullptr: no twiddles
    uint32_t ns, k0, k1;    // Stockham columns of the two columns
    template <bool ADJACENT>  // k1 = k0 + 1, k0 and ns even
    __device__ __forceinline__ cpx2 at(const float2 *t, uint32_t row) const
    {
        const float2 *p = t + static_cast<size_t>(row) * ns + k0;
        if constexpr (ADJACENT) {
            const float4 q = __ldg(reinterpret_cast<const float4 *>(p));
            return pair_of(make_float2(q.x, q.y), make_float2(q.z, q.w));
        } else {
            return pair_of(__ldg(p), __ldg(p - k0 + k1));
        }
    }
    // v[r] *= w0 t2[r][k] of both columns, r < R: w0 = W^(j k), the product W^((j + r NBF) k)
    template <int R, bool FWD, bool ADJACENT>
    __device__ __forceinline__ void apply(cpx2 *v, cpx2 w0) const
    {
        v[0] = cmul(v[0], dir<FWD>(w0));
#pragma unroll
        for (int r = 1; r < R; r++) v[r] = cmul(v[r], dir<FWD>(cmul(w0, at<ADJACENT>(t2, r))));
    }
};

template <class Q, int T, int P, bool FWD>
__device__ __forceinline__ void pair_stage0(cpx2 *v, const float4 *tile, int lane, const PassTwiddle &tw,
                                            const PassTable2 &two)
{
    constexpr int R = Q::r[0], NBF = Q::N / R, NB = (NBF + T - 1) / T;
    static_assert(NBF % T == 0, "every thread owns whole butterflies");
#pragma unroll
    for (int b = 0; b < NB; b++) {
#pragma unroll
        for (int r = 0; r < R; r++) {
            const float4 q = tile[(lane + b * T + r * NBF) * P];
            v[b * R + r] = pair_of(make_float2(q.x, q.y), make_float2(q.z, q.w));
        }
    }
#pragma unroll
    for (int b = 0; b < NB; b++) {
        if (tw.t2) {
            const int j = lane + b * T;
            if (tw.k1 == tw.k0 + 1 && ((tw.k0 | tw.ns) & 1) == 0)
                tw.template apply<R, FWD, true>(
                    v + b * R, tw.t1 ? tw.at<true>(tw.t1, j) : pair_of(two.at(j, tw.k0), two.at(j, tw.k1)));
            else
                tw.template apply<R, FWD, false>(
                    v + b * R, tw.t1 ? tw.at<false>(tw.t1, j) : pair_of(two.at(j, tw.k0), two.at(j, tw.k1)));
        }
        dft<R, FWD>(v + b * R);
    }
}

// Last-stage stores of two columns, element stride es complex values.
struct PairColumns {
    float2 *c0, *c1;
    int64_t es;
    bool second;  // the second column exists
    bool wide;    // the columns are adjacent and every element pair is 16-byte aligned
    template <class Q, int S, int T>
    __device__ __forceinline__ void store(const cpx2 *v, int lane) const
    {
        constexpr int R = Q::r[S], NS = Q::ns(S), NBF = Q::N / R, NB = (NBF + T - 1) / T;
        const int64_t step = NS * es;
#pragma unroll
        for (int b = 0; b < NB; b++) {
            const int64_t at = (lane + b * T) * es;  // last stage: butterfly j writes elements j + r NS
            float2 *p0 = c0 + at, *p1 = c1 + at;
            if (wide) {
#pragma unroll
                for (int r = 0; r < R; r++) st_stream(p0 + r * step, first_of(v[b * R + r]), second_of(v[b * R + r]));
            } else {
#pragma unroll
                for (int r = 0; r < R; r++) st_stream(p0 + r * step, first_of(v[b * R + r]));
                if (second) {
#pragma unroll
                    for (int r = 0; r < R; r++) st_stream(p1 + r * step, second_of(v[b * R + r]));
                }
            }
        }
    }
};

// Last stage with contiguous column outputs (element stride 1, the first pass
// of a multi-pass transform), read with the elements fastest: the threads of a
// warp store runs of at least 16 consecutive elements of a column, where the
// pair-fastest order would store four elements of eight columns (measured on
// 65536 x 256: 86 % of the L1 throughput went into those stores).
template <class Q, int T, int P, int PITCH, bool FWD, class Base>
__device__ __forceinline__ void pair_last_runs(cpx2 *v, const float4 *w, int tid, uint32_t cols, const Base &base,
                                               const float2 *__restrict__ stw)
{
    constexpr int S = Q::S - 1, R = Q::r[S], NS = Q::ns(S), NB = NS * P / (P * T);
    static_assert(NS * P % (P * T) == 0 && NS % 16 == 0, "whole butterflies, runs of 16");
    using Row = typename PairTile<Q, P, PITCH>::template Row<S - 1>;
#pragma unroll
    for (int b = 0; b < NB; b++) {
        const int q = tid + b * P * T, j = q % NS, p = q / NS;
        const Row row{const_cast<float4 *>(w) + p};
#pragma unroll
        for (int r = 0; r < R; r++) v[b * R + r] = row(j + r * NS);
#pragma unroll
        for (int r = 1; r < R; r++)
            v[b * R + r] = cmul(v[b * R + r], dir<FWD>(__ldg(stw + Q::tw_off(S) + (r - 1) * NS + j)));
        dft<R, FWD>(v + b * R);
        if (static_cast<uint32_t>(2 * p) < cols) {
            float2 *c0 = base(2 * p) + j;
#pragma unroll
            for (int r = 0; r < R; r++) st_stream(c0 + r * NS, first_of(v[b * R + r]));
        }
        if (static_cast<uint32_t>(2 * p + 1) < cols) {
            float2 *c1 = base(2 * p + 1) + j;
#pragma unroll
            for (int r = 0; r < R; r++) st_stream(c1 + r * NS, second_of(v[b * R + r]));
        }
    }
}

// Stages S >= 1: gather from the work tile, last stage to `dst`.  The caller's
// barrier separates stage 0's scatter from the first gather here.
template <class Q, int T, int P, bool FWD, int S, class Dst>
__device__ __forceinline__ void pair_stages(cpx2 *v, float4 *w, const Dst &dst, int lane, bool active,
                                            const float2 *__restrict__ stw)
{
    using Tile = PairTile<Q, P>;
    sgather<Q, S, T, FWD>(v, typename Tile::template Row<S - 1>{w}, lane, active, stw);
    if constexpr (S == Q::S - 1) {
        if (active) dst.template store<Q, S, T>(v, lane);
    } else {
        __syncthreads();
        sscatter<Q, S, T>(v, typename Tile::template Row<S>{w}, lane, active);
        __syncthreads();
        pair_stages<Q, T, P, FWD, S + 1>(v, w, dst, lane, active, stw);
    }
}

}  // namespace sipfft
