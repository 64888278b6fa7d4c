// Host walk of the pair tiles' index arithmetic (pair_tile.cuh): every shape that
// pair_shape accepts for a range of lengths, rows and columns, is run through the
// stages of pair_tile_impl.cuh element by element in double, each shared-memory
// word checked against the tile buffer, and the result compared with a direct DFT.
// Built and run by tests/test_pair_tile_model.py (nvcc, CPU only).
#include <cmath>
#include <complex>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "codelets.cuh"
#include "pair_tile.cuh"

using namespace sipfft;
using cd = std::complex<double>;

static std::vector<int> factors(int n, int largest, bool up)
{
    std::vector<int> r;
    while (n > 1) {
        int f = 0;
        for (int k = largest; k >= 2 && !f; k--)
            if (n % k == 0) f = k;
        if (!f) return {};
        r.push_back(f);
        n /= f;
    }
    if (up) r = std::vector<int>(r.rbegin(), r.rend());
    return r;
}

#define CHECK(c) do { if (!(c)) { std::printf("FAILED %s n=%d rows=%d P=%d R0=%d\n", #c, n, d.rows, d.P, d.st[0].R); return false; } } while (0)

static bool run(int n, const std::vector<int> &rad, bool rows, bool runs, int64_t raw_dist, int pairs)
{
    PairDesc d{};
    if (!pair_shape(d, n, rad.data(), static_cast<int>(rad.size()), rows, runs, raw_dist, pairs)) return true;
    CHECK(d.buf_words * 16 <= kPairBufBytes && d.buf_words % 8 == 0 && (rows || ((1 << d.lp) == d.P && kPairThreads % d.P == 0)));
    // staged data: rows (one element in, the worst alignment) and columns
    if (rows)
        CHECK(2 * (int64_t(d.P) * raw_dist) + 1 <= int64_t(d.buf_words) * 2);
    else
        CHECK(int64_t(n) * d.P <= d.buf_words);
    // one of the two transforms of each pair: they share every index
    std::vector<std::vector<cd>> x(d.P, std::vector<cd>(n)), got(d.P, std::vector<cd>(n, cd(1e300, 0)));
    for (int p = 0; p < d.P; p++)
        for (int e = 0; e < n; e++) x[p][e] = cd(std::sin(1.0 + 3.7 * e + p * 1.3), std::cos(0.3 * e * e + p));
    std::vector<cd> work(d.buf_words, cd(1e300, 0));
    for (int s = 0; s < d.nstages; s++) {
        const PairStage &t = d.st[s];
        const bool last = s == d.nstages - 1;
        const bool fast_e = rows || (last && runs && s > 0);
        const int nb = pair_nb(t.R);
        CHECK(t.tasks == t.nbf * d.P && t.tasks <= kPairThreads * nb);
        std::vector<cd> v(size_t(kPairThreads) * nb * t.R);
        std::vector<int> seen(t.tasks, 0);
        for (int phase = 0; phase < 2; phase++)
            for (int tid = 0; tid < kPairThreads; tid++)
                for (int b = 0; b < nb; b++) {
                    const PairTask k0 = fast_e ? pair_task<true>(tid, b, d.lp, t.nbf, t.nbf_m, t.tasks)
                                               : pair_task<false>(tid, b, d.lp, t.nbf, t.nbf_m, t.tasks);
                    const int p = k0.p, j = k0.j;
                    const bool on = k0.on;
                    const int q = s == 0 ? j : static_cast<int>((uint64_t(uint32_t(j)) * t.ns_m) >> 32);
                    CHECK(p >= 0 && p < d.P && j >= 0 && j < t.nbf && q == j / t.ns);
                    cd *a = &v[(size_t(tid) * nb + b) * t.R];
                    if (phase == 0) {
                        if (on) seen[p * t.nbf + j]++;
                        const int k = j - q * t.ns;
                        for (int r = 0; r < t.R; r++) {
                            if (s == 0) {
                                a[r] = x[p][j + r * t.nbf];
                            } else {
                                const int at = pair_gather_at(d.SP, d.SE, t.gpad, p, j, q) + r * t.gstep;
                                CHECK(at >= 0 && at < d.buf_words);
                                a[r] = work[at] * std::polar(1.0, -2 * M_PI * double(r) * k / (double(t.ns) * t.R));
                            }
                        }
                        std::vector<cd> y(t.R);
                        for (int m = 0; m < t.R; m++)
                            for (int r = 0; r < t.R; r++) y[m] += a[r] * std::polar(1.0, -2 * M_PI * double((r * m) % t.R) / t.R);
                        for (int r = 0; r < t.R; r++) a[r] = y[r];
                    } else if (on) {
                        for (int r = 0; r < t.R; r++) {
                            if (last) got[p][j + r * t.ns] = a[r];  // outputs j + r ns (k = j)
                            const int at = pair_scatter_at(d.SP, d.SE, t.spad, t.ns, t.R, p, j, q) + r * t.ns * d.SE;
                            CHECK(at >= 0 && at < d.buf_words);
                            work[at] = a[r];
                        }
                    }
                }
        for (int c : seen) CHECK(c == 1);
    }
    // R2C reads the transform from the work tile in natural order (rows, unpadded last boundary)
    if (rows && d.nstages > 1)
        for (int p = 0; p < d.P; p++)
            for (int e = 0; e < n; e++) CHECK(std::abs(work[p * d.SP + e] - got[p][e]) == 0.0 || (d.nstages == 1));
    for (int p = 0; p < d.P; p += std::max(1, d.P / 2)) {
        double err = 0, ref = 0;
        for (int k = 0; k < n; k += (n > 300 ? 37 : 1)) {
            cd y = 0;
            for (int e = 0; e < n; e++) y += x[p][e] * std::polar(1.0, -2 * M_PI * double((int64_t(e) * k) % n) / n);
            err += std::norm(y - got[p][k]);
            ref += std::norm(y);
        }
        CHECK(err <= 1e-20 * ref * n);
    }
    return true;
}

// Inter-pass twiddles W_F^(e k), e = j + r n / r0, in FP32: the rms error of t1 t2 with t1 from
// the tables of roots less one is not above that of one two-level lookup (two rounded factors).
static bool twiddles(int64_t F, int n, int r0)
{
    auto root = [](int64_t m, int64_t d) {
        const double t = 2 * M_PI * double(m % d) / double(d);
        return make_float2(float(std::cos(t)), float(-std::sin(t)));
    };
    auto less_one = [](int64_t m, int64_t d) {
        const double t = M_PI * double(m % d) / double(d), s = std::sin(t);
        return make_float2(float(-2 * s * s), float(-std::sin(2 * t)));
    };
    int log2l = 1;
    while ((int64_t(1) << (2 * log2l)) < F) log2l++;
    const int64_t L = int64_t(1) << log2l, ns = F / n;
    double lookup = 0, product = 0;
    uint64_t seed = 12345;
    auto draw = [&](int64_t below) {
        seed = seed * 6364136223846793005ull + 1442695040888963407ull;
        return int64_t((seed >> 33) % uint64_t(below));
    };
    for (int i = 0; i < 200000; i++) {
        const int64_t k = draw(ns), j = draw(n / r0), r = draw(r0), m = (j + r * (n / r0)) * k % F, u = j * k;
        const cd exact = std::polar(1.0, -2 * M_PI * double(m) / double(F));
        auto off = [&](float2 w) { return std::norm(cd(w.x, w.y) - exact); };
        const float2 t2 = root(r * k * (n / r0), F);
        lookup += off(cmul(root(m % L, F), root(m / L * L, F)));
        product += off(cmul(root_product(less_one(u % L, F), less_one(u / L * L, F)), t2));
    }
    if (product <= lookup * 1.02) return true;  // (2 %: the spread of 200000 draws)
    std::printf("FAILED twiddles F=%lld n=%d r0=%d: lookup %.3g product %.3g\n", (long long)F, n, r0,
                std::sqrt(lookup / 2e5), std::sqrt(product / 2e5));
    return false;
}

// Relative rms error of the radix-R codelet on two transforms (index 0) and on one (index 1).
template <int R, bool FWD>
static void codelet_errors(double (&e)[2])
{
    double err[2] = {}, ref = 0;
    uint32_t seed = 7;
    auto draw = [&] { return float(((seed = seed * 1664525u + 1013904223u) >> 8) / 8388608.0 - 1.0); };
    for (int t = 0; t < 4000; t++) {
        float2 one[R];
        cpx2 two[R];
        cd x[R];
        for (int i = 0; i < R; i++) {
            one[i].x = draw();
            one[i].y = draw();
            x[i] = cd(one[i].x, one[i].y);
            two[i] = pair_of(make_float2(draw(), draw()), one[i]);
        }
        dft<R, FWD>(one);
        dft<R, FWD>(two);
        for (int k = 0; k < R; k++) {
            cd y = 0;
            for (int j = 0; j < R; j++) y += x[j] * std::polar(1.0, (FWD ? -2 : 2) * M_PI * ((j * k) % R) / R);
            const float2 s = second_of(two[k]);
            err[0] += std::norm(cd(s.x, s.y) - y);
            err[1] += std::norm(cd(one[k].x, one[k].y) - y);
            ref += std::norm(y);
        }
    }
    for (int i = 0; i < 2; i++) e[i] = std::sqrt(err[i] / ref);
}

// Primes and powers of two: the same operations.  Composites: no twiddles on two transforms, and
// fewer roundings (each input passes the products of one twiddle less: at least 4 % of the error).
template <int R>
static bool codelets()
{
    double f[2], b[2];
    codelet_errors<R, true>(f);
    codelet_errors<R, false>(b);
    const bool composite = R == 6 || R == 10 || R == 12 || R == 14 || R == 15;
    const bool ok = composite ? f[0] < 0.96 * f[1] && b[0] < 0.96 * b[1] : f[0] == f[1] && b[0] == b[1];
    if (!ok) std::printf("FAILED radix %d: two %.3g %.3g one %.3g %.3g\n", R, f[0], b[0], f[1], b[1]);
    return ok;
}

int main()
{
    int shapes = 0;
    bool ok = true;
    ok = codelets<2>() && codelets<3>() && codelets<4>() && codelets<5>() && codelets<6>() && codelets<7>() &&
         codelets<8>() && codelets<9>() && codelets<10>() && codelets<11>() && codelets<12>() && codelets<13>() &&
         codelets<14>() && codelets<15>() && codelets<16>();
    ok = twiddles(1 << 25, 256, 16) && twiddles(1 << 27, 512, 16) && twiddles(15625 * 2048, 250, 10) && ok;
    std::vector<int> lengths;
    for (int n = 2; n <= 100; n++) lengths.push_back(n);
    for (int n : {210, 225, 240, 243, 250, 252, 256, 300, 343, 375, 400, 441, 480, 512, 540, 625, 720, 768, 960, 1000,
                  1024, 1080, 1152, 1280, 1331, 1500, 1536, 1792, 1920, 2000, 2048, 2187, 2197})
        lengths.push_back(n);
    for (int n : lengths)
        for (int largest : {16, 10, 7})
            for (int up = 0; up < 2; up++) {
                const std::vector<int> r = factors(n, largest, up != 0);
                if (r.empty()) continue;
                for (int pairs : {32, 11, 8, 5, 4, 3, 1}) {
                    ok = run(n, r, true, false, n, pairs) && run(n, r, true, false, n + 1, pairs) &&
                         run(n, r, false, false, n, pairs) && run(n, r, false, true, n, pairs) && ok;
                    shapes += 4;
                }
            }
    // division by a constant
    for (int64_t v : {1, 2, 3, 5, 7, 64, 100, 127, 1000, 65537, 1 << 20, (1 << 30) + 1, 0x7fffffff})
        for (uint32_t m : {0u, 1u, 2u, 99u, 100u, 65535u, 65536u, 123456789u, 0x3fffffffu, 0x7fffffffu}) {
            const FastDiv f = fast_div(v);
            if (f.div(m) != m / v || f.mod(m) != m % v) {
                std::printf("FAILED division %u / %lld\n", m, (long long)v);
                ok = false;
            }
        }
    // ... up to the last index of a tile that starts at the largest column, by powers of two (the
    // divisors whose reciprocal has the largest error) and their neighbours
    for (int64_t v = 1; v < int64_t(1) << 31; v *= 2)
        for (int64_t w : {v, v - 1, v + 1})
            for (int64_t m = kPairMaxCols - 64; m < kPairMaxCols + 2 * kPairThreads; m++) {
                if (w < 1) continue;
                const FastDiv f = fast_div(w);
                if (f.div(static_cast<uint32_t>(m)) != m / w) {
                    std::printf("FAILED division %lld / %lld\n", (long long)m, (long long)w);
                    ok = false;
                }
            }
    std::printf("%d shapes %s\n", shapes, ok ? "ALL OK" : "FAILED");
    return ok ? 0 : 1;
}
