// Segment and bond passes of the chain sweeps with the y transform split
// between them.
//
// A segment step is an inverse 3-D transform, the segment factor, a forward
// transform and the bond factor.  With m2 = Y1 * Y2 the y transform is done
// half in each of two passes, so that both work on small tiles:
//
//   real-space pass (k_split_real): the Y1 rows y0 + Y2 j (j < Y1) of one x,
//     all z.  DFT over k1 (Y1 values, in registers), z inverse, pointwise op,
//     z forward, DFT over j.  The twiddles w_{m2}^{y0 k1} between the halves
//     are applied here.
//   k-space pass (k_split_k): the Y2 consecutive rows k1 Y2 + y0 (y0 < Y2) of
//     W columns z, all x.  DFT over y0 (Y2 values, in registers), x forward,
//     pointwise op at (kx, ky = k1 + Y1 k2, kz), x inverse, DFT over k2.
//
// Between the passes a field holds, at row y0 + Y2 k1, the half-transformed
// value (y0, k1): each tile of either pass reads and writes the same rows, so
// a pass may run in place.
//
// Each 1-D transform along z (x) is two register butterflies, m = A * B
// (inverse along z: radix A, then B; forward in reversed order, B then A), so
// the op sits between two radix-B butterflies of the same thread and a pass is
// five register phases with four shared-memory exchanges, whatever the length:
//     Y1 | A | B op B | A | Y1      (real space; Y2 | A | B op B | A | Y2)
// (k_cube_k, the k-space pass of the 96 and 128 cubes, has three phases and two
// exchanges.)
//
// Why split: one yz plane per block (k_plane) leaves one block of few warps
// per SM on planes of mixed radix and does not fit at all above 112^2 in
// complex128, where the y transform became two more passes over memory.  The
// tiles here are 8-40 KB (k_cube_k at 128: 74 KB; long extents more, up to the
// 225 KB of a block), so several blocks share an SM and hide each other's loads
// and barriers, and every grid whose extents have two radices takes two passes
// per segment.
// Measured on one B200, whole calls with the plane and line passes of
// passes.cuh and with these, in turn: chain of 50 segments at 128^3 complex128
// 3.56 -> 1.98 ms (72.7 -> 40 us per segment; its six field transfers, one of
// them the stored propagator's, take 31 at the measured copy rate);
// 40 segments at 90 x 125 x 100 complex128 5.28 -> 2.00 ms; step at 96^3
// complex64, N = 32, 8.7 -> 2.1 ms; step at 64^3 complex64, N = 50, 1.44 -> 1.15
// ms.  A pass alone is bound by issue slots and by the latency of its dependent
// phases: at 128^3 complex64 the real-space pass issues 0.41 instructions per
// cycle and scheduler over 22 K active cycles.  In a step graph the passes
// overlap: 101 MB in 20.4 us per segment there, 0.75 of the copy rate.
//
// The radices come from a plan: RtPlan reads them from the geometry (a
// uniform switch per phase; any extents that factor into two radices),
// CubePlan has every size at compile time (real space: the square planes of the
// production cubes with any x extent; k space: the cubes), XPlan the x extents
// 32, 64 and 128.
#pragma once

#include "passes.cuh"

#include <algorithm>
#include <vector>

namespace ftsp {

constexpr int SPLIT_NT = 512;   // largest block
constexpr int SPLIT_NT_HUGE = 256;   // of RtHugePlan
constexpr int SPLIT_RADICES[] = {1, 2, 3, 4, 5, 6, 8, 9, 10, 12, 15, 16, 18, 20, 24, 25, 32};

struct SplitGeom {
    int m1, m2, m3;
    int ok;                  // the extents factor (see split_setup)
    int big_r, big_k;        // passes with radices that need RtBigPlan (1) or RtHugePlan (2)
    // (shorts: four bytes more in this kernel argument shift the parameters after
    // it, and the run-time complex128 passes came out with other registers, steps
    // at 20^3 400 -> 410 us)
    short plane;             // side of the yz plane whose compile-time real-space plan runs, 0: a run-time plan
    short xct;               // x extent whose compile-time k-space plan runs, 0: a run-time plan
    int Y1, Y2;
    // real-space pass: m3 = zA * zB, G row groups (y0 .. y0 + G - 1) per block
    int zA, zB, G, rows;     // rows = G * Y1
    int zA1, zB1;            // padded radices of the two exchanges
    int pn, pa, pb;          // row pitches: natural order, after radix A, after radix B
    int rt, r_threads;       // tile values, threads
    FastDiv fzA, fzB, fm3, fY1;
    // k-space pass: m1 = xA * xB, W columns, C = Y2 * W values per x
    int xA, xB, W, C, pc;
    int kt, k_threads, nzb;
    FastDiv fC, fW, fnzb;
    // twiddle tables: [t * zA + i] = w^(i t) (t < zB), [t * zB + i] (t < zA),
    // the same of x, and [y0 * Y1 + k1] = w_{m2}^(y0 k1)
    const void *tza, *tzb, *txa, *txb, *ty;
    const void* tx;          // w_{m1}^j
};

// ---- factors and layouts (constexpr: compile-time plans evaluate them too) ----
constexpr bool split_radix(int r)
{
    for (int k : SPLIT_RADICES)
        if (k == r) return true;
    return false;
}
// n = a * b, a >= b, as even as possible, a at most amax, b at most bmax
constexpr bool split_pair(int n, int amax, int bmax, int& a, int& b, bool with27 = false)
{
    for (int x = 1; x <= amax; ++x)
        if (n % x == 0 && x * x >= n && n / x <= bmax && (split_radix(x) || (with27 && x == 27)) &&
            (split_radix(n / x) || (with27 && n / x == 27))) {
            a = x;
            b = n / x;
            return true;
        }
    return false;
}
__host__ __device__ constexpr int split_max(int a, int b) { return a > b ? a : b; }
constexpr int split_round32(int t) { return t < 32 ? 32 : (t + 31) / 32 * 32; }
// Extra shared-memory cycles of one access by 64 consecutive threads, thread
// l at value (l / o) * p + (l % o) * q: banks of 8 (complex64) or 16 bytes, 16
// or 8 threads served at a time.
constexpr int bank_cost(int lanes, int banks, int o, int p, int q)
{
    int cost = 0;
    for (int l0 = 0; l0 < lanes && l0 < 64; l0 += banks) {
        int n[16] = {}, worst = 1;
        for (int l = l0; l < lanes && l < l0 + banks; ++l) {
            const int b = ((l / o) * p + (l % o) * q) % banks;
            n[b] += 1;
            worst = split_max(worst, n[b]);
        }
        cost += worst - 1;
    }
    return cost;
}
// Exchange of radix r in a row of n values: written r values apart by the
// (row, i < n / r) threads, read by (row, i < r): padded radix r1, row pitch.
constexpr void split_exchange(int n, int r, int rows, int banks, int& r1, int& pitch)
{
    const int o = n / r;
    int best = 1 << 30;
    for (int pad = r; pad <= r + 1; ++pad)
        for (int p = o * pad; p < o * pad + banks; ++p) {
            const int c = bank_cost(rows * o, banks, o, p, pad) + bank_cost(rows * r, banks, r, p, 1);
            if (c < best) {
                best = c;
                r1 = pad;
                pitch = p;
            }
        }
}

// Tiles of G row groups (real space) and W columns (k space): pitches, sizes,
// threads.
constexpr bool split_tiles(SplitGeom& g, int value_bytes, int G, int W)
{
    const int banks = 128 / value_bytes;
    const int m1 = g.m1, m3 = g.m3;
    g.G = G;
    g.rows = g.G * g.Y1;
    g.r_threads = split_round32(split_max(g.rows * g.zA, g.G * m3));
    if (g.r_threads > 256) g.r_threads = 256;
    int best = 1 << 30;
    for (int p = m3; p < m3 + banks; ++p) {   // natural order: (row, i < B) at row p + i
        const int c = bank_cost(g.rows * g.zB, banks, g.zB, p, 1);
        if (c < best) {
            best = c;
            g.pn = p;
        }
    }
    split_exchange(m3, g.zA, g.rows, banks, g.zA1, g.pa);
    split_exchange(m3, g.zB, g.rows, banks, g.zB1, g.pb);
    g.rt = g.rows * split_max(g.pn, split_max(g.pa, g.pb));
    g.fzA = make_fastdiv(g.zA); g.fzB = make_fastdiv(g.zB); g.fm3 = make_fastdiv(m3); g.fY1 = make_fastdiv(g.Y1);
    g.W = W;
    g.C = g.Y2 * g.W;
    g.k_threads = split_round32(split_max(g.C * g.xA, m1 * g.W));
    const int most = g.big_k == 2 ? SPLIT_NT_HUGE : SPLIT_NT;
    if (g.k_threads > most) g.k_threads = most;
    best = 1 << 30;
    for (int p = g.C; p < g.C + banks; ++p) {
        const int c = bank_cost(64, banks, g.W, p, 1) + bank_cost(64, banks, g.C, p, 1) +
                      bank_cost(64, banks, g.C, g.xA * p, 1) + bank_cost(64, banks, g.C, g.xB * p, 1);
        if (c < best) {
            best = c;
            g.pc = p;
        }
    }
    g.kt = m1 * g.pc;
    // both buffers of both passes within the shared memory of a block
    if ((2LL * g.rt + 2 * m3 + g.rows) * value_bytes > 225 * 1024 || (2LL * g.kt + 2 * m1) * value_bytes > 225 * 1024) return false;
    g.nzb = (m3 + g.W - 1) / g.W;
    g.fC = make_fastdiv(g.C); g.fW = make_fastdiv(g.W); g.fnzb = make_fastdiv(g.nzb);
    return true;
}

constexpr bool split_setup(SplitGeom& g, int m1, int m2, int m3, int value_bytes)
{
    g.m1 = m1; g.m2 = m2; g.m3 = m3;
    g.ok = 0;
    const bool square = m2 == m3 && (m3 == 32 || m3 == 48 || m3 == 64 || m3 == 96 || m3 == 128);
    g.big_k = 0;
    // the butterfly pair around the op (radix B) holds the op's operands
    // beside its values: 10 at most, except in RtBigPlan and RtHugePlan
    if (!split_pair(m3, 16, 10, g.zA, g.zB) || !split_pair(m1, 16, 10, g.xA, g.xB) || !split_pair(m2, 16, 16, g.Y1, g.Y2)) {
        if (!split_pair(m3, 32, 16, g.zA, g.zB) || !split_pair(m1, 32, 16, g.xA, g.xB) || !split_pair(m2, 32, 16, g.Y1, g.Y2)) {
            // two radices above 16, or 27, along x only, where the real-space
            // pass has a compile-time plan (steps with N = 16, with it and with
            // the run-time passes: 243 x 32 x 32 complex64 0.78 and 2.5 ms, 640 x
            // 64 x 64 complex128 7.3 and 13.6)
            if (!square || !split_pair(m3, 16, 10, g.zA, g.zB) || !split_pair(m1, 32, 32, g.xA, g.xB, true) ||
                !split_pair(m2, 16, 16, g.Y1, g.Y2))
                return false;
            g.big_k = 2;
        } else if (g.Y1 > 16) {   // the long half of y in the pass whose tiles are narrower
            const int t = g.Y1;
            g.Y1 = g.Y2;
            g.Y2 = t;
        }
    }
    // compile-time plans: the square planes of the production cubes, with any x
    // extent; the x extents of the cubes, with their plane or (32, 64, 128) any
    // rows of 4 or 8 and whole tiles.  128 x 8 in complex64 has half the threads
    // of the run-time plan and pays beside a run-time real-space pass only where
    // its blocks cover the SMs (steps with N = 16, run-time and this plan: 64
    // blocks, 128 x 64 x 32, 745 and 870 us; 135 blocks, 128 x 72 x 60, 985 and
    // 1039; 200 blocks, 128 x 80 x 80, 1507 and 1295)
    g.plane = square ? m3 : 0;
    const bool few = m1 == 128 && g.Y2 == 8 && value_bytes == 8 && !square && g.Y1 * (m3 / 4) < 148;
    g.xct = g.plane == m1 ? m1 : (m1 == 32 || m1 == 64 || m1 == 128) && (g.Y2 == 4 || g.Y2 == 8) && m3 % 4 == 0 && !few ? m1 : 0;
    // real space: as many row groups per block as leave two blocks per SM
    int G = 1;
    for (int t = 2; t <= g.Y2 && !g.plane; ++t)
        if (g.Y2 % t == 0 && m1 * (g.Y2 / t) >= 296 && t * g.Y1 * m3 <= 1024 && t * split_max(g.Y1 * g.zA, m3) <= 256) G = t;
    // k space: 32 bytes of every row (one memory sector)
    int W = split_max(1, 32 / value_bytes);
    while (W > 1 && (W / 2 >= m3 || (long long)m1 * g.Y2 * W * value_bytes > 72 * 1024)) W /= 2;
    g.big_r = g.zA > 16 || g.zB > 10 || g.Y1 > 16;
    if (!g.big_k) g.big_k = g.xA > 16 || g.xB > 10 || g.Y2 > 16;
    // narrower tiles of a long x
    while (!split_tiles(g, value_bytes, G, W)) {
        if (W == 1) return false;
        W /= 2;
    }
    g.ok = 1;
    return true;
}

// ---- plans ----
// RtPlan takes everything from the geometry argument, gives a thread one
// butterfly per phase and exchanges between two buffers (one barrier each).
struct RtPlan {
    static constexpr bool CT = false, PLANE = false;
    static constexpr bool INPLACE = false;
    static constexpr SplitGeom G = SplitGeom{};
    static constexpr int RNT = 256, KNT = SPLIT_NT;
    static constexpr int AMAX = 16, BMAX = 10;
    // blocks per SM asked of the compiler, real space and k space
    template <typename T> static constexpr int rmin = sizeof(T) == 4 ? 3 : 2;
};
// The same for lengths that need a radix of 18 to 32 (125 = 25 x 5, 320 = 20 x
// 16) or two large radices (192 = 16 x 12): its own kernels, so that the others
// keep their registers.
struct RtBigPlan : RtPlan {
    static constexpr int AMAX = 32, BMAX = 16;
    template <typename T> static constexpr int rmin = 1;
};
// The k-space pass of x extents with two radices above 16 or one of 27 (486 = 27
// x 18, 640 = 32 x 20): a thread holds up to 32 points and the op's operands, so
// blocks are half as large.
struct RtHugePlan : RtPlan {
    static constexpr int KNT = SPLIT_NT_HUGE;
    static constexpr int AMAX = 33, BMAX = 33;
    template <typename T> static constexpr int rmin = 1;
};
// A cube of N points a side at compile time.  One buffer: a phase reads,
// synchronises and writes.  Where the radix-B (and Y2) butterflies are a
// multiple of the others in number, a thread takes several of them.
constexpr int split_nt(int base, int a, int b)   // threads: a phase of `base` butterflies and two more
{
    const int nt = split_round32(base);
    return a % nt == 0 && b % nt == 0 ? nt : split_round32(split_max(base, split_max(a, b)));
}
constexpr SplitGeom split_box(int m1, int n, int value_bytes)   // m1 planes of n x n points
{
    SplitGeom g{};
    split_setup(g, m1, n, n, value_bytes);
    g.r_threads = split_nt(split_max(g.rows * g.zB, g.G * n), g.rows * g.zA, g.rows * g.zA);
    g.k_threads = split_nt(g.C * g.xB, g.C * g.xA, m1 * g.W);
    return g;
}
constexpr SplitGeom split_cube(int n, int value_bytes) { return split_box(n, n, value_bytes); }
// The real-space pass takes it for any number of N x N planes (it uses m1 for
// nothing but its grid).
template <int N, typename T>
struct CubePlan {
    static constexpr bool CT = true, PLANE = true;
    static constexpr bool INPLACE = true;
    static constexpr SplitGeom G = split_cube(N, 2 * (int)sizeof(T));
    static constexpr int RNT = G.r_threads, KNT = G.k_threads;
    static constexpr int AMAX = 16, BMAX = 10;
    template <typename T2> static constexpr int rmin = 1;
    static_assert(G.G == 1, "one row group per block on every grid with this plane");
};
// The k-space pass of m1 = X points along x and rows of Y2 = 4 or 8 at compile
// time, m2, m3 and Y1 from the geometry argument (m3 a multiple of the tile
// width).
template <int X, int Y2, typename T>
struct XPlan {
    static constexpr bool CT = true, PLANE = false;
    static constexpr bool INPLACE = true;
    // Threads: as in the cubes, but a thread per butterfly of the widest phase
    // where a thread had four of a phase or 256 bytes of values (steps with
    // N = 16, the cubes' rule and this one: 128 x 32 x 32 complex64 617 and 384
    // us, complex128 739 and 571, 128 x 64 x 64 complex128 1225 and 1026; the
    // others lose by it: 128 x 64 x 64 complex64 736 and 849, 32 x 64 x 64 344
    // and 362)
    static constexpr SplitGeom threads(SplitGeom g)
    {
        const int nt = g.k_threads, widest = split_max(g.C * g.xA, g.m1 * g.W);
        const int rows = (g.m1 * g.W + nt - 1) / nt, mid = (g.C * g.xA + nt - 1) / nt;
        const int values = split_max(split_max(rows * g.Y2, mid * g.xB), (g.C * g.xB + nt - 1) / nt * g.xA);
        if (split_max(rows, mid) >= 4 || values * 2 * (int)sizeof(T) >= 256) g.k_threads = split_round32(widest);
        return g;
    }
    static constexpr SplitGeom G = threads(split_box(X, Y2 == 4 ? 32 : 64, 2 * (int)sizeof(T)));
    static constexpr int RNT = G.r_threads, KNT = G.k_threads;
    static constexpr int AMAX = 16, BMAX = 10;
    template <typename T2> static constexpr int rmin = 1;
    static_assert(G.Y2 == Y2 && G.m1 == X, "representative grid");
};

// Values of the twiddle tables, in the order tza, tzb, txa, txb, ty, tx
// (2 m3 + 3 m1 + m2 values); tw(n, j) gives exp(-2 pi i j / n).
template <class V, class Tw>
inline std::vector<V> split_tables(const SplitGeom& g, Tw tw)
{
    std::vector<V> t;
    auto put = [&](int n, int inner, int outer) {
        for (int o = 0; o < outer; ++o)
            for (int i = 0; i < inner; ++i) t.push_back(tw(n, (o * i) % n));
    };
    put(g.m3, g.zA, g.zB);
    put(g.m3, g.zB, g.zA);
    put(g.m1, g.xA, g.xB);
    put(g.m1, g.xB, g.xA);
    put(g.m2, g.Y1, g.Y2);
    for (int j = 0; j < g.m1; ++j) t.push_back(tw(g.m1, j));
    return t;
}
template <class V>
inline void split_point_tables(SplitGeom& g, const V* base)
{
    g.tza = base;
    g.tzb = base + g.m3;
    g.txa = base + 2 * g.m3;
    g.txb = base + 2 * g.m3 + g.m1;
    g.ty = base + 2 * g.m3 + 2 * g.m1;
    g.tx = base + 2 * g.m3 + 2 * g.m1 + g.m2;
}
template <class P, class V>
inline size_t split_real_smem(const SplitGeom& g)
{
    return std::max(sizeof(V) * (size_t)((P::INPLACE ? 1 : 2) * g.rt + 2 * g.m3 + g.rows), (size_t)4096);
}
template <class P, class V>
inline size_t split_k_smem(const SplitGeom& g)
{
    return std::max(sizeof(V) * (size_t)((P::INPLACE ? 1 : 2) * g.kt + 2 * g.m1), (size_t)4096);
}

// ---- device ----
// 9 = 3 x 3 with the twiddles w9, w9^2, w9^4
template <int S, typename V>
__device__ __forceinline__ void dft9(V* u)
{
    using R = typename RealOf<V>::type;
    const R c1 = R(0.76604444311897803520239265055541668), s1 = R(0.64278760968653932632264340990726344);   // 40 degrees
    const R c2 = R(0.17364817766693034885171662676931480), s2 = R(0.98480775301220805936674302458952302);   // 80 degrees
    const R c4 = R(-0.93969262078590838405410927732473147), s4 = R(0.34202014332566873304409961468225958);  // 160 degrees
    auto rot = [](V z, R c, R sn) { return mkc<V>(z.x * c - S * z.y * sn, z.y * c + S * z.x * sn); };
    V a[3][3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
#pragma unroll
        for (int k = 0; k < 3; ++k) a[j][k] = u[j + 3 * k];
        dft3<S>(a[j]);
    }
    a[1][1] = rot(a[1][1], c1, s1);
    a[1][2] = rot(a[1][2], c2, s2);
    a[2][1] = rot(a[2][1], c2, s2);
    a[2][2] = rot(a[2][2], c4, s4);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        V b[3] = {a[0][k], a[1][k], a[2][k]};
        dft3<S>(b);
        u[k] = b[0];
        u[k + 3] = b[1];
        u[k + 6] = b[2];
    }
}

template <int S, int R, typename V>
__device__ __forceinline__ void dft_factor(V* u)
{
    if constexpr (R == 9) dft9<S>(u);
    else dftR<S, R>(u);
}

// Composite butterflies.  Coprime factors need no twiddles: with inputs
// n = (Q n1 + P n2) mod PQ and outputs k = k1 mod P, k2 mod Q (the prime-factor
// algorithm), the transform is P-point DFTs over n1 and Q-point ones over n2.
template <int S, int P, int Q, typename V>
__device__ __forceinline__ void dft_coprime(V* u)
{
    constexpr int N = P * Q;
    V a[N];
#pragma unroll
    for (int n2 = 0; n2 < Q; ++n2) {
        V b[P];
#pragma unroll
        for (int n1 = 0; n1 < P; ++n1) b[n1] = u[(Q * n1 + P * n2) % N];
        dft_factor<S, P>(b);
#pragma unroll
        for (int k1 = 0; k1 < P; ++k1) a[k1 * Q + n2] = b[k1];
    }
#pragma unroll
    for (int k1 = 0; k1 < P; ++k1) {
        V b[Q];
#pragma unroll
        for (int n2 = 0; n2 < Q; ++n2) b[n2] = a[k1 * Q + n2];
        dft_factor<S, Q>(b);
#pragma unroll
        for (int k = 0; k < N; ++k)
            if (k % P == k1) u[k] = b[k % Q];
    }
}

// 25 = 5 x 5 with the twiddles w25^(j k)
template <int S, typename V>
__device__ __forceinline__ void dft25(V* u)
{
    using R = typename RealOf<V>::type;
    // cos and sin of 2 pi j / 25 for the products j = 1 .. 16
    constexpr double c[17] = {1.0, 0.96858316112863108148, 0.87630668004386363938, 0.72896862742141157547, 0.53582679497899660946,
                              0.30901699437494742410, 0.06279051952931337608, -0.18738131458572463066, -0.42577929156507266490,
                              -0.63742398974868967902, -0.80901699437494742410, -0.92977648588825144064, -0.99211470131447776388,
                              -0.99211470131447776388, -0.92977648588825144064, -0.80901699437494742410, -0.63742398974868967902};
    constexpr double sn[17] = {0.0, 0.24868988716485478824, 0.48175367410171529046, 0.68454710592868869210, 0.84432792550201508508,
                               0.95105651629515357212, 0.99802672842827155733, 0.98228725072868865924, 0.90482705246601951990,
                               0.77051324277578920853, 0.58778525229247312917, 0.36812455268467797320, 0.12533323356430427018,
                               -0.12533323356430427018, -0.36812455268467797320, -0.58778525229247312917, -0.77051324277578920853};
    V a[5][5];
#pragma unroll
    for (int j = 0; j < 5; ++j) {
#pragma unroll
        for (int k = 0; k < 5; ++k) a[j][k] = u[j + 5 * k];
        dft5<S>(a[j]);
#pragma unroll
        for (int k = 1; k < 5; ++k)
            if (j > 0) {
                const R cc = R(c[j * k]), ss = R(sn[j * k]);
                const V z = a[j][k];
                a[j][k] = mkc<V>(z.x * cc - S * z.y * ss, z.y * cc + S * z.x * ss);
            }
    }
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        V b[5] = {a[0][k], a[1][k], a[2][k], a[3][k], a[4][k]};
        dft5<S>(b);
#pragma unroll
        for (int t = 0; t < 5; ++t) u[k + 5 * t] = b[t];
    }
}

// 27 = 9 x 3 with the twiddles w27^(j k)
template <int S, typename V>
__device__ __forceinline__ void dft27(V* u)
{
    using R = typename RealOf<V>::type;
    // cos and sin of 2 pi j / 27 for the products j = 0 .. 16
    constexpr double c[17] = {1.0, 0.97304487057982383883, 0.89363264032341224819, 0.7660444431189780352,
                              0.59715859170278616485, 0.3960797660391568237, 0.17364817766693034885,
                              -0.058144828910475828539, -0.2868032327110902531, -0.5, -0.68624163786873358573,
                              -0.83548781141293641965, -0.93969262078590838405, -0.99323835774194298855,
                              -0.99323835774194298855, -0.93969262078590838405, -0.83548781141293641965};
    constexpr double sn[17] = {0.0, 0.23061587074244017845, 0.44879918020046217279, 0.64278760968653932632,
                               0.80212319275504378508, 0.91821610688027401476, 0.98480775301220805937,
                               0.99830815827126820805, 0.95798951231548887444, 0.86602540378443864676,
                               0.72737364157304869599, 0.54950897807080603526, 0.34202014332566873304,
                               0.11609291412523022968, -0.11609291412523022968, -0.34202014332566873304,
                               -0.54950897807080603526};
    V a[3][9];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
#pragma unroll
        for (int k = 0; k < 9; ++k) a[j][k] = u[j + 3 * k];
        dft9<S>(a[j]);
#pragma unroll
        for (int k = 1; k < 9; ++k)
            if (j > 0) a[j][k] = crot<S>(a[j][k], R(c[j * k]), R(sn[j * k]));
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        V b[3] = {a[0][k], a[1][k], a[2][k]};
        dft3<S>(b);
#pragma unroll
        for (int t = 0; t < 3; ++t) u[k + 9 * t] = b[t];
    }
}

// cos(2 pi m / 32)
__host__ __device__ constexpr double cos32(int m)
{
    constexpr double c[9] = {1.0, 0.98078528040323044913, 0.92387953251128675613, 0.83146961230254523708, 0.70710678118654752440,
                             0.55557023301960222474, 0.38268343236508977173, 0.19509032201612826785, 0.0};
    m &= 31;
    if (m > 16) m = 32 - m;
    return m <= 8 ? c[m] : -c[16 - m];
}
// 32 = 4 x 8: DFT8 over the stride-4 sub-sequences, twiddles w32^(j k), DFT4
template <int S, typename V>
__device__ __forceinline__ void dft32(V* u)
{
    using R = typename RealOf<V>::type;
    V a[4][8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
#pragma unroll
        for (int k = 0; k < 8; ++k) a[j][k] = u[j + 4 * k];
        dft8<S>(a[j]);
#pragma unroll
        for (int k = 1; k < 8; ++k) {
            if (j == 0) continue;
            if (j * k == 8) {
                a[j][k] = mul_si<S>(a[j][k]);
            } else {
                const R c = R(cos32(j * k)), sn = R(cos32(j * k + 24));   // sin(t) = cos(t - 90 degrees)
                const V z = a[j][k];
                a[j][k] = mkc<V>(z.x * c - S * z.y * sn, z.y * c + S * z.x * sn);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        V b[4] = {a[0][k], a[1][k], a[2][k], a[3][k]};
        dft4<S>(b);
#pragma unroll
        for (int t = 0; t < 4; ++t) u[k + 8 * t] = b[t];
    }
}

template <int S, int R, typename V>
__device__ __forceinline__ void dft_any(V* u)
{
    if constexpr (R == 6) dft_coprime<S, 2, 3>(u);
    else if constexpr (R == 9) dft9<S>(u);
    else if constexpr (R == 10) dft_coprime<S, 2, 5>(u);
    else if constexpr (R == 12) dft_coprime<S, 4, 3>(u);
    else if constexpr (R == 15) dft_coprime<S, 3, 5>(u);
    else if constexpr (R == 18) dft_coprime<S, 2, 9>(u);
    else if constexpr (R == 20) dft_coprime<S, 4, 5>(u);
    else if constexpr (R == 24) dft_coprime<S, 8, 3>(u);
    else if constexpr (R == 25) dft25<S>(u);
    else if constexpr (R == 27) dft27<S>(u);
    else if constexpr (R == 32) dft32<S>(u);
    else dftR<S, R>(u);
}

template <int R>
struct RadixTag {
    static constexpr int value = R;
};
// f(RadixTag<r>) for the radix of a phase: CTR at compile time, r (uniform
// over the grid, at most MAX) at run time
template <bool CT, int CTR, int MAX, class F>
__device__ __forceinline__ void by_radix(int r, F&& f)
{
    if constexpr (CT) {
        f(RadixTag<CTR>{});
    } else {
        switch (r) {
        case 1: f(RadixTag<1>{}); break;
        case 2: f(RadixTag<2>{}); break;
        case 3: f(RadixTag<3>{}); break;
        case 4: f(RadixTag<4>{}); break;
        case 5: f(RadixTag<5>{}); break;
        case 6: f(RadixTag<6>{}); break;
        case 8: f(RadixTag<8>{}); break;
        case 9: f(RadixTag<9>{}); break;
        case 10: f(RadixTag<10>{}); break;
        default:
            if constexpr (MAX > 10) {
                if (r == 12) f(RadixTag<12>{});
                else if (r == 15) f(RadixTag<15>{});
                else if (r == 16) f(RadixTag<16>{});
            }
            if constexpr (MAX > 16) {
                if (r == 18) f(RadixTag<18>{});
                else if (r == 20) f(RadixTag<20>{});
                else if (r == 24) f(RadixTag<24>{});
                else if (r == 25) f(RadixTag<25>{});
                else if (r == 32) f(RadixTag<32>{});
            }
            if constexpr (MAX > 32) {
                if (r == 27) f(RadixTag<27>{});
            }
            break;
        }
    }
}

template <int S, int R, typename V>
__device__ __forceinline__ void twiddle_table(V* u, const V* tab, int stride)
{
#pragma unroll
    for (int t = 1; t < R; ++t) {
        V w = tab[t * stride];
        if (S > 0) w.y = -w.y;
        u[t] = cmul(u[t], w);
    }
}

// One phase: `items` butterflies of radix R over the block, gather(idx, u) then
// finish(idx, u), and a barrier at the end where SYNC.  At compile time (ITEMS,
// NT threads) a thread gathers all of its butterflies first, with the in-place
// barrier after them.
template <class P, int R, int ITEMS, int NT, bool INPLACE, bool SYNC, typename V, class Ga, class Fi>
__device__ __forceinline__ void split_phase(int items, Ga gather, Fi finish)
{
    if constexpr (P::CT) {
        constexpr int NB = (ITEMS + NT - 1) / NT;
        V u[NB][R];
#pragma unroll
        for (int q = 0; q < NB; ++q) {
            const int idx = threadIdx.x + q * NT;
            if (ITEMS % NT == 0 || idx < ITEMS) gather(idx, u[q]);
        }
        if (INPLACE) __syncthreads();
#pragma unroll
        for (int q = 0; q < NB; ++q) {
            const int idx = threadIdx.x + q * NT;
            if (ITEMS % NT == 0 || idx < ITEMS) finish(idx, u[q]);
        }
    } else {
        static_assert(P::CT || !INPLACE, "the run-time plan exchanges between two buffers");
#pragma unroll 1
        for (int idx = threadIdx.x; idx < items; idx += blockDim.x) {
            V u[R];
            gather(idx, u);
            finish(idx, u);
        }
    }
    if (SYNC) __syncthreads();
}

// geometry member: a constant of the plan, or the kernel argument's
#define FTSP_PL(m) (P::CT ? P::G.m : g.m)
// the same of the members that depend on the yz plane
#define FTSP_PP(m) (P::PLANE ? P::G.m : g.m)
// quotient by a geometry member with its magic-number divisor
#define FTSP_DIV(i, m, f) (P::CT ? (int)((unsigned)(i) / (unsigned)split_max(1, P::G.m)) : (int)fdiv(i, g.f))

// registers a thread is given: at 128^3 complex64 ops with one operand per
// point fit 72 (7 blocks of 128 threads: 1024 blocks in one wave; 20.4 us per
// segment with its bond pass, 21.0 with 128 registers), and 64^3 steps are
// faster with it too (22.4 against 24.1 ms per 20 steps); on the mixed-radix
// cubes and at 32^3, 128 registers keep more loads in flight (96^3 17.4 -> 16.5
// us per segment with its share of the pair densities, 48^3 6.2 -> 5.8, 32^3
// 5.1 -> 4.9)
template <typename T, class Op>
constexpr int split_regs(int n)
{
    return sizeof(T) == 4 && (n == 128 || n == 64) ? (op_loads<Op>::value == 0 ? 64 : op_loads<Op>::value == 1 ? 72 : 96) : 128;
}
template <class P, typename T, class Op>
constexpr int split_min_blocks(int nt)
{
    // small complex128 cubes never fill an SM: no cap (32^3: 4.9 us per segment
    // in the step graph, 5.4 capped at 128)
    if (P::CT && sizeof(T) == 8 && P::G.m1 <= 64) return 1;
    return P::CT ? split_max(1, 65536 / (nt * split_regs<T, Op>(P::G.m1))) : nt <= 256 ? P::template rmin<T> : 1;
}

// Real-space pass: grid (m1 * Y2 / G, fields).
template <typename T, class P, int S1, int S2, class Op>
__global__ void __launch_bounds__(P::RNT, split_min_blocks<P, T, Op>(P::RNT))
    k_split_real(SplitGeom g, const cplx<T>* src, cplx<T>* dst, size_t fstride, Op op)
{
    using V = cplx<T>;
    constexpr int NT = P::RNT;
    constexpr bool IP = P::INPLACE;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int m2 = FTSP_PL(m2), m3 = FTSP_PL(m3), Y1 = FTSP_PL(Y1), Y2 = FTSP_PL(Y2), zA = FTSP_PL(zA), zB = FTSP_PL(zB);
    const int rows = FTSP_PL(rows), pn = FTSP_PL(pn), pa = FTSP_PL(pa), pb = FTSP_PL(pb), zA1 = FTSP_PL(zA1), zB1 = FTSP_PL(zB1);
    const int gpb = FTSP_PL(G), rt = FTSP_PL(rt);
    const int nthr = P::CT ? NT : (int)blockDim.x;
    V* b0 = reinterpret_cast<V*>(smem_raw);
    V* b1 = IP ? b0 : b0 + rt;
    V* ta = b1 + rt;       // radix B stage of butterfly i < A
    V* tb = ta + m3;       // radix A stage of butterfly i < B
    V* ty = tb + m3;       // [group][k1]
    const int tid = threadIdx.x;
    const int nyb = Y2 / gpb;
    const int f = blockIdx.y;
    const int x = blockIdx.x / nyb;
    const int y0 = (blockIdx.x - x * nyb) * gpb;
    const size_t base = (size_t)f * fstride + (size_t)x * m2 * m3;
    for (int j = tid; j < m3; j += nthr) {
        ta[j] = reinterpret_cast<const V*>(g.tza)[j];
        tb[j] = reinterpret_cast<const V*>(g.tzb)[j];
    }
    for (int j = tid; j < rows; j += nthr) ty[j] = reinterpret_cast<const V*>(g.ty)[y0 * Y1 + j];
    pdl_wait();
    // every block has started once all have come here: the next pass may take
    // what is idle and run its prologue (it waits for this one before it
    // touches a field)
    pdl_trigger();
    op_preload(op);
    if constexpr (S1 != 0) {
        __syncthreads();   // twiddles
        by_radix<P::CT, P::G.Y1, P::AMAX>(Y1, [&](auto rc) {
            constexpr int R = decltype(rc)::value;
            split_phase<P, R, P::G.G * P::G.m3, NT, false, true, V>(gpb * m3,
                [&](int idx, V (&u)[R]) {
                    const int gr = FTSP_DIV(idx, m3, fm3), z = idx - gr * m3;
                    const V* s = src + base + (size_t)(y0 + gr) * m3 + z;
                    const size_t st = (size_t)Y2 * m3;
#pragma unroll
                    for (int t = 0; t < R; ++t) u[t] = s[t * st];
                },
                [&](int idx, V (&u)[R]) {
                    const int gr = FTSP_DIV(idx, m3, fm3), z = idx - gr * m3;
                    if (y0 + gr) twiddle_table<S1, R>(u, ty + gr * R, 1);
                    dft_any<S1, R>(u);
                    V* d = b0 + gr * R * pn + z;
#pragma unroll
                    for (int t = 0; t < R; ++t) d[t * pn] = u[t];
                });
        });
        by_radix<P::CT, P::G.zA, P::AMAX>(zA, [&](auto rc) {
            constexpr int R = decltype(rc)::value;
            split_phase<P, R, P::G.rows * P::G.zB, NT, IP, false, V>(rows * zB,
                [&](int idx, V (&u)[R]) {
                    const int r = FTSP_DIV(idx, zB, fzB), i = idx - r * zB;
                    const V* s = b0 + r * pn + i;
#pragma unroll
                    for (int t = 0; t < R; ++t) u[t] = s[t * zB];
                },
                [&](int idx, V (&u)[R]) {
                    const int r = FTSP_DIV(idx, zB, fzB), i = idx - r * zB;
                    dft_any<S1, R>(u);
                    V* d = b1 + r * pa + i * zA1;
#pragma unroll
                    for (int t = 0; t < R; ++t) d[t] = u[t];
                });
        });
    }
    op.begin();
    __syncthreads();
    by_radix<P::CT, P::G.zB, P::BMAX>(zB, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        // one operand per point: a butterfly's loads are in flight across the
        // gather; wider ops load a few points at a time
        constexpr int CH = op_loads<Op>::value <= 1 ? R : (R < 4 ? R : sizeof(T) == 4 ? 4 : 2);
        auto place = [&](int idx, int& r, int& i, int& y, size_t& off) {
            r = FTSP_DIV(idx, zA, fzA);
            i = idx - r * zA;
            const int gr = FTSP_DIV(r, Y1, fY1), j = r - gr * Y1;
            y = y0 + gr + Y2 * j;
            off = base + (size_t)y * m3 + i;
        };
        auto gather = [&](int idx, V (&u)[R]) {
            const int r = FTSP_DIV(idx, zA, fzA), i = idx - r * zA;
#pragma unroll
            for (int t = 0; t < R; ++t) u[t] = S1 != 0 ? b1[r * pa + i + t * zA1] : mkc<V>(T(0), T(0));
        };
        auto loads = [&](int idx, typename Op::Pre (&pre)[CH]) {
            int r, i, y;
            size_t off;
            place(idx, r, i, y, off);
#pragma unroll
            for (int t = 0; t < CH; ++t) pre[t] = op.load(f, off + t * zA);
        };
        auto finish = [&](int idx, V (&u)[R], typename Op::Pre (&pre)[CH]) {
            int r, i, y;
            size_t off;
            place(idx, r, i, y, off);
            if constexpr (S1 != 0) {
                twiddle_table<S1, R>(u, ta + i, zA);
                dft_any<S1, R>(u);
            }
#pragma unroll
            for (int t = 0; t < R; ++t) {
                if constexpr (CH < R) {
                    if (t % CH == 0) {
#pragma unroll
                        for (int k = 0; k < CH; ++k)
                            if (t + k < R) pre[k] = op.load(f, off + (t + k) * zA);
                    }
                }
                u[t] = op.apply(f, x, y, i + t * zA, off + t * zA, u[t], pre[t % CH]);
            }
        };
        auto scatter = [&](int idx, V (&u)[R]) {
            if constexpr (S2 != 0) {
                const int r = FTSP_DIV(idx, zA, fzA), i = idx - r * zA;
                dft_any<S2, R>(u);
                V* d = b0 + r * pb + i * zB1;
#pragma unroll
                for (int t = 0; t < R; ++t) d[t] = u[t];
            }
        };
        typename Op::Pre pre[CH];
        if constexpr (P::CT) {
            constexpr int ITEMS = P::G.rows * P::G.zA;
            constexpr int NB = (ITEMS + NT - 1) / NT;
            V u[NB][R];
            auto valid = [&](int idx) { return ITEMS % NT == 0 || idx < ITEMS; };
            if constexpr (CH == R) {
                if (valid(tid)) loads(tid, pre);
            }
#pragma unroll
            for (int q = 0; q < NB; ++q)
                if (valid(tid + q * NT)) gather(tid + q * NT, u[q]);
            if (IP && S1 != 0 && S2 != 0) __syncthreads();
#pragma unroll
            for (int q = 0; q < NB; ++q) {
                const int idx = tid + q * NT;
                if (valid(idx)) {
                    finish(idx, u[q], pre);
                    if constexpr (CH == R) {
                        if (q + 1 < NB && valid(idx + NT)) loads(idx + NT, pre);
                    }
                    scatter(idx, u[q]);
                }
            }
        } else {
#pragma unroll 1
            for (int idx = tid; idx < rows * zA; idx += blockDim.x) {
                V u[R];
                if constexpr (CH == R) loads(idx, pre);
                gather(idx, u);
                finish(idx, u, pre);
                scatter(idx, u);
            }
        }
    });
    if constexpr (S2 != 0) {
        __syncthreads();
        by_radix<P::CT, P::G.zA, P::AMAX>(zA, [&](auto rc) {
            constexpr int R = decltype(rc)::value;
            split_phase<P, R, P::G.rows * P::G.zB, NT, IP, true, V>(rows * zB,
                [&](int idx, V (&u)[R]) {
                    const int r = FTSP_DIV(idx, zB, fzB), i = idx - r * zB;
                    const V* s = b0 + r * pb + i;
#pragma unroll
                    for (int t = 0; t < R; ++t) u[t] = s[t * zB1];
                },
                [&](int idx, V (&u)[R]) {
                    const int r = FTSP_DIV(idx, zB, fzB), i = idx - r * zB;
                    twiddle_table<S2, R>(u, tb + i, zB);
                    dft_any<S2, R>(u);
                    V* d = b1 + r * pn + i;
#pragma unroll
                    for (int t = 0; t < R; ++t) d[t * zB] = u[t];
                });
        });
        by_radix<P::CT, P::G.Y1, P::AMAX>(Y1, [&](auto rc) {
            constexpr int R = decltype(rc)::value;
            split_phase<P, R, P::G.G * P::G.m3, NT, false, false, V>(gpb * m3,
                [&](int idx, V (&u)[R]) {
                    const int gr = FTSP_DIV(idx, m3, fm3), z = idx - gr * m3;
                    const V* s = b1 + gr * R * pn + z;
#pragma unroll
                    for (int t = 0; t < R; ++t) u[t] = s[t * pn];
                },
                [&](int idx, V (&u)[R]) {
                    const int gr = FTSP_DIV(idx, m3, fm3), z = idx - gr * m3;
                    dft_any<S2, R>(u);
                    if (y0 + gr) twiddle_table<S2, R>(u, ty + gr * R, 1);
                    V* d = dst + base + (size_t)(y0 + gr) * m3 + z;
                    const size_t st = (size_t)Y2 * m3;
#pragma unroll
                    for (int t = 0; t < R; ++t) d[t * st] = u[t];
                });
        });
    }
    op.end(reinterpret_cast<double*>(b0), blockIdx.x + (size_t)blockIdx.y * gridDim.x);
}

// k-space pass: grid (Y1 * nzb, fields); the input of field f is field
// op_src_field(op, f) of src.  Without the second transform (S2 = 0) the op
// stores, in natural order.
template <typename T, class P, int S1, int S2, class Op>
__global__ void __launch_bounds__(P::KNT, split_min_blocks<P, T, Op>(P::KNT))
    k_split_k(SplitGeom g, const cplx<T>* src, cplx<T>* dst, size_t fstride, Op op)
{
    using V = cplx<T>;
    constexpr int NT = P::KNT;
    constexpr bool IP = P::INPLACE;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int m1 = FTSP_PL(m1), m2 = FTSP_PP(m2), m3 = FTSP_PP(m3), Y1 = FTSP_PP(Y1), Y2 = FTSP_PL(Y2), xA = FTSP_PL(xA), xB = FTSP_PL(xB);
    const int W = FTSP_PL(W), C = FTSP_PL(C), pc = FTSP_PL(pc), kt = FTSP_PL(kt), nzb = FTSP_PP(nzb);
    const int nthr = P::CT ? NT : (int)blockDim.x;
    V* b0 = reinterpret_cast<V*>(smem_raw);
    V* b1 = IP ? b0 : b0 + kt;
    V* ta = b1 + kt;
    V* tb = ta + m1;
    const int tid = threadIdx.x;
    const int f = blockIdx.y;
    const int k1 = P::PLANE ? (int)(blockIdx.x / (unsigned)split_max(1, P::G.nzb)) : (int)fdiv(blockIdx.x, g.fnzb);
    const int z0 = (blockIdx.x - k1 * nzb) * W;
    const size_t plane = (size_t)m2 * m3;
    const size_t inner = (size_t)k1 * Y2 * m3 + z0;
    const V* sp = src + (size_t)op_src_field(op, f) * fstride + inner;
    V* dp = dst + (size_t)f * fstride + inner;
    const size_t fbase = (size_t)f * fstride;
    // the last tile of a row may be partial
    const bool whole = P::CT ? !P::PLANE || P::G.m3 % split_max(1, P::G.W) == 0 : false;
    for (int j = tid; j < m1; j += nthr) {
        ta[j] = reinterpret_cast<const V*>(g.txa)[j];
        tb[j] = reinterpret_cast<const V*>(g.txb)[j];
    }
    pdl_wait();
    pdl_trigger();   // as in the real-space pass
    by_radix<P::CT, P::G.Y2, P::AMAX>(Y2, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        split_phase<P, R, P::G.m1 * P::G.W, NT, false, true, V>(m1 * W,
            [&](int idx, V (&u)[R]) {
                const int x = FTSP_DIV(idx, W, fW), w = idx - x * W;
                const bool in = whole || z0 + w < m3;
                const V* s = sp + (size_t)x * plane + w;
#pragma unroll
                for (int t = 0; t < R; ++t) u[t] = in ? s[(size_t)t * m3] : mkc<V>(T(0), T(0));
            },
            [&](int idx, V (&u)[R]) {
                const int x = FTSP_DIV(idx, W, fW), w = idx - x * W;
                dft_any<S1, R>(u);
                V* d = b0 + x * pc + w;
#pragma unroll
                for (int t = 0; t < R; ++t) d[t * W] = u[t];
            });
    });
    by_radix<P::CT, P::G.xA, P::AMAX>(xA, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        split_phase<P, R, P::G.C * P::G.xB, NT, IP, false, V>(C * xB,
            [&](int idx, V (&u)[R]) {
                const int i = FTSP_DIV(idx, C, fC), c = idx - i * C;
                const V* s = b0 + i * pc + c;
#pragma unroll
                for (int t = 0; t < R; ++t) u[t] = s[t * xB * pc];
            },
            [&](int idx, V (&u)[R]) {
                const int i = FTSP_DIV(idx, C, fC), c = idx - i * C;
                dft_any<S1, R>(u);
                V* d = b1 + i * xA * pc + c;
#pragma unroll
                for (int t = 0; t < R; ++t) d[t * pc] = u[t];
            });
    });
    op.begin();
    __syncthreads();
    by_radix<P::CT, P::G.xB, P::BMAX>(xB, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        split_phase<P, R, P::G.C * P::G.xA, NT, IP, true, V>(C * xA,
            [&](int idx, V (&u)[R]) {
                const int i = FTSP_DIV(idx, C, fC), c = idx - i * C;
                const V* s = b1 + i * pc + c;
#pragma unroll
                for (int t = 0; t < R; ++t) u[t] = s[t * xA * pc];
            },
            [&](int idx, V (&u)[R]) {
                const int i = FTSP_DIV(idx, C, fC), c = idx - i * C;
                const int k2 = FTSP_DIV(c, W, fW), w = c - k2 * W;
                const int y = k1 + Y1 * k2;
                const size_t off = fbase + (size_t)i * plane + (size_t)y * m3 + z0 + w;
                twiddle_table<S1, R>(u, ta + i, xA);
                dft_any<S1, R>(u);
                if (whole || z0 + w < m3) {
                    typename Op::Pre pre[R];
#pragma unroll
                    for (int t = 0; t < R; ++t) pre[t] = op.load(f, off + (size_t)t * xA * plane);
#pragma unroll
                    for (int t = 0; t < R; ++t)
                        u[t] = op.apply(f, i + t * xA, y, z0 + w, off + (size_t)t * xA * plane, u[t], pre[t]);
                }
                if constexpr (S2 != 0) {
                    dft_any<S2, R>(u);
                    V* d = b0 + i * xB * pc + c;
#pragma unroll
                    for (int t = 0; t < R; ++t) d[t * pc] = u[t];
                }
            });
    });
    if constexpr (S2 != 0) {
        by_radix<P::CT, P::G.xA, P::AMAX>(xA, [&](auto rc) {
            constexpr int R = decltype(rc)::value;
            split_phase<P, R, P::G.C * P::G.xB, NT, IP, true, V>(C * xB,
                [&](int idx, V (&u)[R]) {
                    const int i = FTSP_DIV(idx, C, fC), c = idx - i * C;
                    const V* s = b0 + i * pc + c;
#pragma unroll
                    for (int t = 0; t < R; ++t) u[t] = s[t * xB * pc];
                },
                [&](int idx, V (&u)[R]) {
                    const int i = FTSP_DIV(idx, C, fC), c = idx - i * C;
                    twiddle_table<S2, R>(u, tb + i, xB);
                    dft_any<S2, R>(u);
                    V* d = b1 + i * pc + c;
#pragma unroll
                    for (int t = 0; t < R; ++t) d[t * xB * pc] = u[t];
                });
        });
        by_radix<P::CT, P::G.Y2, P::AMAX>(Y2, [&](auto rc) {
            constexpr int R = decltype(rc)::value;
            split_phase<P, R, P::G.m1 * P::G.W, NT, false, false, V>(m1 * W,
                [&](int idx, V (&u)[R]) {
                    const int x = FTSP_DIV(idx, W, fW), w = idx - x * W;
                    const V* s = b1 + x * pc + w;
#pragma unroll
                    for (int t = 0; t < R; ++t) u[t] = s[t * W];
                },
                [&](int idx, V (&u)[R]) {
                    const int x = FTSP_DIV(idx, W, fW), w = idx - x * W;
                    dft_any<S2, R>(u);
                    V* d = dp + (size_t)x * plane + w;
                    if (whole || z0 + w < m3) {
#pragma unroll
                        for (int t = 0; t < R; ++t) d[(size_t)t * m3] = u[t];
                    }
                });
        });
    }
    op.end(reinterpret_cast<double*>(b0), blockIdx.x + (size_t)blockIdx.y * gridDim.x);
}

#undef FTSP_PL
#undef FTSP_PP
#undef FTSP_DIV

// The k-space pass of a cube with m1 = XP * XQ in two exchanges instead of
// four (128^3 complex64: 24.0 K -> 17.3 K active cycles, with its real-space
// pass 26.5 -> 20.4 us per segment; 64-byte rows 23.3, 32-byte rows 24.6 with
// the pair densities' share; the smaller cubes have too few threads for it): a thread first holds the Y2 rows of XP points x = i + XQ p of one
// column (DFT over the rows, DFT over p, twiddle), then the XQ points of one
// (p, row, column) for the second x stage, the op and its inverse; it writes
// those back where it read them, so the pass has two barriers and the XP - 1
// twiddles of a thread stay in registers.  About 32 values per thread.
template <int N, typename T>
struct CubeK {
    static constexpr SplitGeom G = split_cube(N, 2 * (int)sizeof(T));
    static constexpr int BANKS = 128 / (2 * (int)sizeof(T));
    static constexpr int XP = N % 3 == 0 ? 3 : 4, XQ = N / XP;
    static constexpr int Y1 = G.Y1, Y2 = G.Y2;
    static constexpr int W = 64 / (2 * (int)sizeof(T));   // columns per tile
    static constexpr int C = Y2 * W;
    static constexpr int PITCH = C + ((W - C) % BANKS + BANKS) % BANKS;    // threads (i, w) on different banks
    static constexpr int NZB = N / W;
    static constexpr int NT = split_round32(split_max(XQ * W, XP * C));
    static constexpr size_t SMEM = 2 * sizeof(T) * (size_t)N * PITCH + 16 * (size_t)N;   // tile, x factors
    static_assert(N % W == 0 && XP * XQ == N, "tile shape");
};

template <typename T, int N, int S1, int S2, class Op>
__global__ void __launch_bounds__(CubeK<N, T>::NT, split_max(1, 65536 / (CubeK<N, T>::NT * (sizeof(T) == 4 ? 128 : 255))))
    k_cube_k(const cplx<T>* __restrict__ tx, const cplx<T>* src, cplx<T>* dst, size_t fstride, Op op)
{
    using V = cplx<T>;
    using P = CubeK<N, T>;
    constexpr int XP = P::XP, XQ = P::XQ, Y1 = P::Y1, Y2 = P::Y2, W = P::W, C = P::C, PITCH = P::PITCH;
    static_assert(S1 != 0 && S2 != 0, "both transforms");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V* tile = reinterpret_cast<V*>(smem_raw);
    const int tid = threadIdx.x;
    const int f = blockIdx.y;
    const int k1 = blockIdx.x / P::NZB;
    const int z0 = (blockIdx.x % P::NZB) * W;
    constexpr size_t plane = (size_t)N * N;
    const size_t inner = (size_t)k1 * Y2 * N + z0;
    const size_t fbase = (size_t)f * fstride;
    const V* sp = src + (size_t)op_src_field(op, f) * fstride + inner;
    V* dp = dst + fbase + inner;
    const int i = tid / W, w = tid % W;
    const bool one = XQ * W == P::NT || tid < XQ * W;
    // the op's x factors: 32 loads per thread from global memory throttled the
    // load queue (2.5 of 9.5 cycles per instruction at 128^3 complex64)
    constexpr bool XTAB = op_has_xtab<Op>::value;
    typename op_xval<Op>::type* xtab = reinterpret_cast<typename op_xval<Op>::type*>(tile + N * PITCH);
    if constexpr (XTAB)
        for (int j = tid; j < N; j += P::NT) xtab[j] = op.x_value(j);
    V tw[XP];
    if (one) {
#pragma unroll
        for (int p = 1; p < XP; ++p) tw[p] = tx[i * p];
    }
    pdl_wait();
    pdl_trigger();
    if (one) {
        V u[XP][Y2];
        const V* s = sp + (size_t)i * plane + w;
#pragma unroll
        for (int p = 0; p < XP; ++p)
#pragma unroll
            for (int y = 0; y < Y2; ++y) u[p][y] = s[(size_t)(p * XQ) * plane + y * N];
#pragma unroll
        for (int p = 0; p < XP; ++p) dft_any<S1, Y2>(u[p]);
        V* d = tile + i * PITCH + w;
#pragma unroll
        for (int y = 0; y < Y2; ++y) {
            V b[XP];
#pragma unroll
            for (int p = 0; p < XP; ++p) b[p] = u[p][y];
            dft_any<S1, XP>(b);
#pragma unroll
            for (int p = 0; p < XP; ++p) {
                if (p > 0) b[p] = cmul(b[p], S1 > 0 ? mkc<V>(tw[p].x, -tw[p].y) : tw[p]);
                d[p * XQ * PITCH + y * W] = b[p];
            }
        }
    }
    op.begin();
    __syncthreads();
    if (XP * C == P::NT || tid < XP * C) {
        const int p = tid / C, c = tid % C;
        const int y = k1 + Y1 * (c / W), z = z0 + c % W;
        const size_t off = fbase + (size_t)p * plane + (size_t)y * N + z;
        V* d = tile + p * XQ * PITCH + c;
        V u[XQ];
#pragma unroll
        for (int q = 0; q < XQ; ++q) u[q] = d[q * PITCH];
        dft_any<S1, XQ>(u);
        constexpr int CH = op_loads<Op>::value == 0 ? XQ : XQ < 4 ? XQ : 4;   // operands in flight
        typename Op::Pre pre[CH];
        typename op_xval<Op>::column col{};
        if constexpr (XTAB) col = op.column(f, y, z);
#pragma unroll
        for (int q = 0; q < XQ; ++q) {
            if (q % CH == 0) {
#pragma unroll
                for (int k = 0; k < CH; ++k)
                    if (q + k < XQ) pre[k] = op.load(f, off + (size_t)(XP * (q + k)) * plane);
            }
            if constexpr (XTAB)
                u[q] = op.apply_x(f, p + XP * q, y, z, off + (size_t)(XP * q) * plane, u[q], pre[q % CH], xtab[p + XP * q], col);
            else
                u[q] = op.apply(f, p + XP * q, y, z, off + (size_t)(XP * q) * plane, u[q], pre[q % CH]);
        }
        dft_any<S2, XQ>(u);
#pragma unroll
        for (int q = 0; q < XQ; ++q) d[q * PITCH] = u[q];
    }
    __syncthreads();
    if (one) {
        V u[XP][Y2];
        const V* s = tile + i * PITCH + w;
#pragma unroll
        for (int y = 0; y < Y2; ++y) {
            V b[XP];
#pragma unroll
            for (int p = 0; p < XP; ++p) {
                b[p] = s[p * XQ * PITCH + y * W];
                if (p > 0) b[p] = cmul(b[p], S2 > 0 ? mkc<V>(tw[p].x, -tw[p].y) : tw[p]);
            }
            dft_any<S2, XP>(b);
#pragma unroll
            for (int p = 0; p < XP; ++p) u[p][y] = b[p];
        }
        V* d = dp + (size_t)i * plane + w;
#pragma unroll
        for (int p = 0; p < XP; ++p) {
            dft_any<S2, Y2>(u[p]);
#pragma unroll
            for (int y = 0; y < Y2; ++y) d[(size_t)(p * XQ) * plane + y * N] = u[p][y];
        }
    }
    op.end(reinterpret_cast<double*>(tile), blockIdx.x + (size_t)blockIdx.y * gridDim.x);
}

// ---- launches ----
// Launched as dependents of the kernel before them (programmatic dependent
// launch): the prologue overlaps its tail.
template <class... Params, class... Args>
inline cudaError_t split_launch(void (*kernel)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t stream, Args... args)
{
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}
template <class P, typename T, int S1, int S2, class Op>
cudaError_t split_real_plan(const SplitGeom& g, const cplx<T>* src, cplx<T>* dst, size_t fstride, int nf, const Op& op,
                            cudaStream_t stream)
{
    const SplitGeom& p = P::CT ? P::G : g;
    return split_launch(k_split_real<T, P, S1, S2, Op>, dim3(g.m1 * (p.Y2 / p.G), nf), p.r_threads,
                        split_real_smem<P, cplx<T>>(p), stream, g, src, dst, fstride, op);
}
template <class P, typename T, int S1, int S2, class Op>
cudaError_t split_k_plan(const SplitGeom& g, const cplx<T>* src, cplx<T>* dst, size_t fstride, int nf, const Op& op,
                         cudaStream_t stream)
{
    const SplitGeom& p = P::CT ? P::G : g;
    SplitGeom a = g;
    if (P::CT) {   // its tile width, not the one of the run-time plans
        a.nzb = g.m3 / p.W;
        a.fnzb = make_fastdiv(a.nzb);
    }
    return split_launch(k_split_k<T, P, S1, S2, Op>, dim3(g.Y1 * a.nzb, nf), p.k_threads, split_k_smem<P, cplx<T>>(p),
                        stream, a, src, dst, fstride, op);
}
// blocks of one field of the real-space pass
inline int split_real_blocks(const SplitGeom& g) { return g.m1 * (g.Y2 / g.G); }

// The planes and x extents of the production cubes run their compile-time plans
// (where g says so); the k-space half of the plain transforms is run-time.
template <typename T, int S1, int S2, class Op>
cudaError_t split_real_launch(const SplitGeom& g, const cplx<T>* src, cplx<T>* dst, size_t fstride, int nf, const Op& op,
                              cudaStream_t stream)
{
    switch (g.plane) {
        case 32: return split_real_plan<CubePlan<32, T>, T, S1, S2>(g, src, dst, fstride, nf, op, stream);
        case 48: return split_real_plan<CubePlan<48, T>, T, S1, S2>(g, src, dst, fstride, nf, op, stream);
        case 64: return split_real_plan<CubePlan<64, T>, T, S1, S2>(g, src, dst, fstride, nf, op, stream);
        case 96: return split_real_plan<CubePlan<96, T>, T, S1, S2>(g, src, dst, fstride, nf, op, stream);
        case 128: return split_real_plan<CubePlan<128, T>, T, S1, S2>(g, src, dst, fstride, nf, op, stream);
        default: break;
    }
    if (g.big_r) return split_real_plan<RtBigPlan, T, S1, S2>(g, src, dst, fstride, nf, op, stream);
    return split_real_plan<RtPlan, T, S1, S2>(g, src, dst, fstride, nf, op, stream);
}
template <int N, typename T, int S1, int S2, class Op>
cudaError_t cube_k(const SplitGeom& g, const cplx<T>* src, cplx<T>* dst, size_t fstride, int nf, const Op& op, cudaStream_t stream)
{
    using P = CubeK<N, T>;
    return split_launch(k_cube_k<T, N, S1, S2, Op>, dim3(P::Y1 * P::NZB, nf), P::NT, P::SMEM, stream,
                        reinterpret_cast<const cplx<T>*>(g.tx), src, dst, fstride, op);
}
template <typename T, int S1, int S2, class Op>
cudaError_t split_k_launch(const SplitGeom& g, const cplx<T>* src, cplx<T>* dst, size_t fstride, int nf, const Op& op,
                           cudaStream_t stream)
{
    if constexpr (S1 != 0 && S2 != 0) {
        if (g.plane == g.xct) switch (g.xct) {   // cubes
            case 32: return split_k_plan<CubePlan<32, T>, T, S1, S2>(g, src, dst, fstride, nf, op, stream);
            case 48: return split_k_plan<CubePlan<48, T>, T, S1, S2>(g, src, dst, fstride, nf, op, stream);
            case 64: return split_k_plan<CubePlan<64, T>, T, S1, S2>(g, src, dst, fstride, nf, op, stream);
            case 96: return cube_k<96, T, S1, S2>(g, src, dst, fstride, nf, op, stream);
            case 128: return cube_k<128, T, S1, S2>(g, src, dst, fstride, nf, op, stream);
            default: break;
        }
        if (g.xct && g.Y2 == 4) switch (g.xct) {
            case 32: return split_k_plan<XPlan<32, 4, T>, T, S1, S2>(g, src, dst, fstride, nf, op, stream);
            case 64: return split_k_plan<XPlan<64, 4, T>, T, S1, S2>(g, src, dst, fstride, nf, op, stream);
            case 128: return split_k_plan<XPlan<128, 4, T>, T, S1, S2>(g, src, dst, fstride, nf, op, stream);
            default: break;
        }
        if (g.xct && g.Y2 == 8) switch (g.xct) {
            case 32: return split_k_plan<XPlan<32, 8, T>, T, S1, S2>(g, src, dst, fstride, nf, op, stream);
            case 64: return split_k_plan<XPlan<64, 8, T>, T, S1, S2>(g, src, dst, fstride, nf, op, stream);
            case 128: return split_k_plan<XPlan<128, 8, T>, T, S1, S2>(g, src, dst, fstride, nf, op, stream);
            default: break;
        }
    }
    if constexpr (S1 != 0 && S2 == 0) {
        if (g.plane == g.xct) switch (g.xct) {
            case 96: return split_k_plan<CubePlan<96, T>, T, S1, S2>(g, src, dst, fstride, nf, op, stream);
            case 128: return split_k_plan<CubePlan<128, T>, T, S1, S2>(g, src, dst, fstride, nf, op, stream);
            default: break;
        }
    }
    if (g.big_k == 2) return split_k_plan<RtHugePlan, T, S1, S2>(g, src, dst, fstride, nf, op, stream);
    if (g.big_k) return split_k_plan<RtBigPlan, T, S1, S2>(g, src, dst, fstride, nf, op, stream);
    return split_k_plan<RtPlan, T, S1, S2>(g, src, dst, fstride, nf, op, stream);
}

// The sweeps' passes are compiled in split_real_*.cu and split_k_*.cu.
#define FTSP_SPLIT_REAL(PRE, T, S1, S2, KIND)                                                                             \
    PRE cudaError_t split_real_launch<T, S1, S2, OpProp<T, KIND>>(const SplitGeom&, const cplx<T>*, cplx<T>*, size_t, int, \
                                                                  const OpProp<T, KIND>&, cudaStream_t);
#define FTSP_SPLIT_REAL_ALL(PRE, T)                                                                                  \
    FTSP_SPLIT_REAL(PRE, T, 0, -1, FWD_START)                                                                        \
    FTSP_SPLIT_REAL(PRE, T, 1, -1, FWD_MID)                                                                          \
    FTSP_SPLIT_REAL(PRE, T, 1, 0, FWD_LAST)                                                                          \
    FTSP_SPLIT_REAL(PRE, T, 0, 0, FWD_SINGLE)                                                                        \
    FTSP_SPLIT_REAL(PRE, T, 0, 1, BWD_START)                                                                         \
    FTSP_SPLIT_REAL(PRE, T, -1, 1, BWD_MID)                                                                          \
    FTSP_SPLIT_REAL(PRE, T, -1, 0, BWD_LAST)                                                                         \
    FTSP_SPLIT_REAL(PRE, T, 0, 0, BWD_SINGLE)
#define FTSP_SPLIT_K(PRE, T, S1, S2, F, ST)                                                                              \
    PRE cudaError_t split_k_launch<T, S1, S2, OpBond<T, F, ST>>(const SplitGeom&, const cplx<T>*, cplx<T>*, size_t, int, \
                                                                const OpBond<T, F, ST>&, cudaStream_t);
#define FTSP_SPLIT_K_ALL(PRE, T)                                                                                     \
    FTSP_SPLIT_K(PRE, T, -1, 1, true, false)                                                                         \
    FTSP_SPLIT_K(PRE, T, 1, -1, false, true)                                                                         \
    FTSP_SPLIT_K(PRE, T, 1, -1, false, false)
#ifndef FTSP_SPLIT_INSTANCES
FTSP_SPLIT_REAL_ALL(extern template, float)
FTSP_SPLIT_REAL_ALL(extern template, double)
FTSP_SPLIT_K_ALL(extern template, float)
FTSP_SPLIT_K_ALL(extern template, double)
#endif

}  // namespace ftsp
