// FFT pass kernels with fused pointwise work: the run-time plans for grids
// that the split-y passes (split_passes.cuh) do not take, and the ops of both.
//
// A 3-D transform of an m1 x m2 x m3 row-major grid (z fastest) is split
// into passes that each read and write HBM once:
//   * plane pass   : one x-plane (m2 x m3) per CTA, z- and y-transforms in
//                    shared memory (used when the plane fits a block: 227
//                    KB and 512 threads of 32 or 16 values);
//   * z-line pass  : B contiguous z-rows per CTA;
//   * strided pass : an n x W tile of lines along y or x, W contiguous
//                    z-columns wide, so every load and store is a W-element
//                    contiguous run.
// Each kernel is  [load -> transform(S1)] -> pointwise Op -> [transform(S2)
// -> store] -> Op::end (block reductions, reusing the tile as scratch);
// S = 0 skips that transform, -1/+1 select its sign.  The Op sees
// the element's coordinates (in k-space after a transform) and its global
// offset, so propagator, density, stress and smoothing work rides in the same
// pass as the FFT instead of costing extra HBM round trips.
#pragma once

#include "fft_core.cuh"

#include <type_traits>

namespace ftsp {

// Programmatic dependent launch: a pass launched with the programmatic
// stream-serialisation attribute starts while the previous kernel drains;
// griddepcontrol.wait holds it until that kernel has completed and its
// writes are visible, so only the prologue (constant twiddles into shared
// memory, index set-up) overlaps.  launch_dependents lets the next kernel be
// scheduled: the split passes call it as soon as their own wait is over, the
// others once a block has issued its last global reads.  Both are no-ops for
// launches without the attribute.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }


struct PlaneGeom {
    int m1, m2, m3;
    int P;                 // shared-memory pitch of a plane row (m3 + 1)
    const FftPlan1* py;    // device-memory plans of the y and z transforms
    const FftPlan1* pz;
    FastDiv fm2, fm3;
};

struct LineGeom {
    int m1, m2, m3;
    int n;                 // transform length (m1 for x, m2 for y, m3 for z)
    int W;                 // z-columns per tile (strided passes)
    int B;                 // rows per tile (z-line pass)
    int P;                 // shared-memory pitch
    const FftPlan1* p;     // device-memory plan of the transform
    FastDiv fW, fB, fm2, fm3;
};

// ---- block reductions (deterministic: fixed shuffle/smem order) ----
template <int K>
__device__ __forceinline__ void block_sum(double (&v)[K], double* scratch)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int c = 0; c < K; ++c) {
        double x = v[c];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        v[c] = x;
    }
    __syncthreads();
    if (lane == 0) {
#pragma unroll
        for (int c = 0; c < K; ++c) scratch[warp * K + c] = v[c];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int c = 0; c < K; ++c) {
            double s = 0.0;
            for (int w = 0; w < nw; ++w) s += scratch[w * K + c];
            v[c] = s;
        }
    }
    __syncthreads();
}

// ---------------------------------------------------------------------------
// Plane pass: grid (m1, nfields), one x-plane per CTA.
// Shared memory: tile[m2][P] + twiddles(m2) + twiddles(m3).
// ---------------------------------------------------------------------------
template <typename T, int E, int S1, int S2, class Op>
__global__ void __launch_bounds__(1024, 1) k_plane(PlaneGeom g, const cplx<T>* src, cplx<T>* dst,
                                                size_t fstride, const cplx<T>* __restrict__ twy,
                                                const cplx<T>* __restrict__ twz, Op op)
{
    using V = cplx<T>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V* tile = reinterpret_cast<V*>(smem_raw);
    V* sty = tile + (size_t)g.m2 * g.P;
    V* stz = sty + g.m2;
    const int x = blockIdx.x;
    const int f = blockIdx.y;
    const int ne = g.m2 * g.m3;
    const size_t base = (size_t)f * fstride + (size_t)x * ne;
    if (S1 != 0 || S2 != 0) {
        load_twiddles(sty, twy, g.m2);
        load_twiddles(stz, twz, g.m3);
    }
    if (S1 != 0) {
        for (int e0 = threadIdx.x; e0 < ne; e0 += 4 * blockDim.x) {
            V v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int e = e0 + u * blockDim.x;
                if (e < ne) v[u] = src[base + e];
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int e = e0 + u * blockDim.x;
                if (e < ne) {
                    const int y = fdiv(e, g.fm3), z = e - y * g.m3;
                    tile[y * g.P + z] = v[u];
                }
            }
        }
        __syncthreads();
        fft_tile<V, S1, E>(tile, stz, g.pz, g.m2, g.fm2, 1, g.P);
        fft_tile<V, S1, E>(tile, sty, g.py, g.m3, g.fm3, g.P, 1);
    } else {
        __syncthreads();
    }
    op.begin();
    constexpr int PB = sizeof(T) == 4 ? 8 : 4;
    for (int e0 = threadIdx.x; e0 < ne; e0 += PB * blockDim.x) {
        typename Op::Pre pre[PB];
#pragma unroll
        for (int k = 0; k < PB; ++k) {
            const int e = e0 + k * blockDim.x;
            if (e < ne) pre[k] = op.load(f, base + e);
        }
#pragma unroll
        for (int k = 0; k < PB; ++k) {
            const int e = e0 + k * blockDim.x;
            if (e < ne) {
                const int y = fdiv(e, g.fm3), z = e - y * g.m3;
                V v = S1 != 0 ? tile[y * g.P + z] : mkc<V>(T(0), T(0));
                v = op.apply(f, x, y, z, base + e, v, pre[k]);
                if (S2 != 0) tile[y * g.P + z] = v;
            }
        }
    }
    if (S2 != 0) {
        __syncthreads();
        fft_tile<V, S2, E>(tile, stz, g.pz, g.m2, g.fm2, 1, g.P);
        fft_tile<V, S2, E>(tile, sty, g.py, g.m3, g.fm3, g.P, 1);
        for (int e = threadIdx.x; e < ne; e += blockDim.x) {
            const int y = fdiv(e, g.fm3), z = e - y * g.m3;
            dst[base + e] = tile[y * g.P + z];
        }
    }
    op.end(reinterpret_cast<double*>(tile), blockIdx.x + (size_t)blockIdx.y * gridDim.x);
}

// ---------------------------------------------------------------------------
// z-line pass: grid (m1*m2/B, nfields); B rows of m3 per CTA.
// Shared memory: tile[B][P] (P = m3 + 1) + twiddles(m3).
// ---------------------------------------------------------------------------
template <typename T, int E, int S1, int S2, class Op>
__global__ void __launch_bounds__(256, 2) k_zline(LineGeom g, const cplx<T>* src, cplx<T>* dst,
                                                size_t fstride, const cplx<T>* __restrict__ twz, Op op)
{
    using V = cplx<T>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V* tile = reinterpret_cast<V*>(smem_raw);
    V* st = tile + (size_t)g.B * g.P;
    const int f = blockIdx.y;
    const int ne = g.B * g.m3;
    const int row0 = blockIdx.x * g.B;
    const size_t base = (size_t)f * fstride + (size_t)row0 * g.m3;
    if (S1 != 0 || S2 != 0) load_twiddles(st, twz, g.m3);
    if (S1 != 0) {
        for (int e = threadIdx.x; e < ne; e += blockDim.x) {
            const int b = fdiv(e, g.fm3), z = e - b * g.m3;
            tile[b * g.P + z] = src[base + e];
        }
        __syncthreads();
        fft_tile<V, S1, E>(tile, st, g.p, g.B, g.fB, 1, g.P);
    } else {
        __syncthreads();
    }
    op.begin();
    constexpr int PB = sizeof(T) == 4 ? 8 : 4;
    for (int e0 = threadIdx.x; e0 < ne; e0 += PB * blockDim.x) {
        typename Op::Pre pre[PB];
#pragma unroll
        for (int k = 0; k < PB; ++k) {
            const int e = e0 + k * blockDim.x;
            if (e < ne) pre[k] = op.load(f, base + e);
        }
#pragma unroll
        for (int k = 0; k < PB; ++k) {
            const int e = e0 + k * blockDim.x;
            if (e < ne) {
                const int b = fdiv(e, g.fm3), z = e - b * g.m3;
                const int row = row0 + b;
                const int x = fdiv(row, g.fm2), y = row - x * g.m2;
                V v = S1 != 0 ? tile[b * g.P + z] : mkc<V>(T(0), T(0));
                v = op.apply(f, x, y, z, base + e, v, pre[k]);
                if (S2 != 0) tile[b * g.P + z] = v;
            }
        }
    }
    if (S2 != 0) {
        __syncthreads();
        fft_tile<V, S2, E>(tile, st, g.p, g.B, g.fB, 1, g.P);
        for (int e = threadIdx.x; e < ne; e += blockDim.x) {
            const int b = fdiv(e, g.fm3), z = e - b * g.m3;
            dst[base + e] = tile[b * g.P + z];
        }
    }
    op.end(reinterpret_cast<double*>(tile), blockIdx.x + (size_t)blockIdx.y * gridDim.x);
}

// ---------------------------------------------------------------------------
// Strided pass along y (DIM = 1) or x (DIM = 0): grid (outer * m3/W, nf).
// Tile[n][W] (pitch W) of lines; the outer index is x for DIM 1, y for DIM 0.
// ---------------------------------------------------------------------------
template <typename T, int E, int DIM, int S1, int S2, class Op>
__global__ void __launch_bounds__(256, 2) k_strided(LineGeom g, const cplx<T>* src, cplx<T>* dst,
                                                  size_t fstride, const cplx<T>* __restrict__ tw, Op op)
{
    using V = cplx<T>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V* tile = reinterpret_cast<V*>(smem_raw);
    V* st = tile + (size_t)g.n * g.W;
    const int nzb = g.m3 / g.W;
    const int outer = blockIdx.x / nzb;
    const int z0 = (blockIdx.x - outer * nzb) * g.W;
    const int f = blockIdx.y;
    const size_t plane = (size_t)g.m2 * g.m3;
    const size_t lstride = DIM == 1 ? (size_t)g.m3 : plane;
    const size_t base = (size_t)f * fstride + (DIM == 1 ? (size_t)outer * plane : (size_t)outer * g.m3) + z0;
    const int ne = g.n * g.W;
    if (S1 != 0 || S2 != 0) load_twiddles(st, tw, g.n);
    if (S1 != 0) {
        for (int e0 = threadIdx.x; e0 < ne; e0 += 4 * blockDim.x) {
            V v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int e = e0 + u * blockDim.x;
                if (e < ne) {
                    const int j = fdiv(e, g.fW), w = e - j * g.W;
                    v[u] = src[base + j * lstride + w];
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int e = e0 + u * blockDim.x;
                if (e < ne) tile[e] = v[u];
            }
        }
        __syncthreads();
        fft_tile<V, S1, E>(tile, st, g.p, g.W, g.fW, g.W, 1);
    } else {
        __syncthreads();
    }
    op.begin();
    constexpr int PB = sizeof(T) == 4 ? 8 : 4;
    for (int e0 = threadIdx.x; e0 < ne; e0 += PB * blockDim.x) {
        typename Op::Pre pre[PB];
#pragma unroll
        for (int k = 0; k < PB; ++k) {
            const int e = e0 + k * blockDim.x;
            if (e < ne) {
                const int j = fdiv(e, g.fW), w = e - j * g.W;
                pre[k] = op.load(f, base + j * lstride + w);
            }
        }
#pragma unroll
        for (int k = 0; k < PB; ++k) {
            const int e = e0 + k * blockDim.x;
            if (e < ne) {
                const int j = fdiv(e, g.fW), w = e - j * g.W;
                const int x = DIM == 1 ? outer : j;
                const int y = DIM == 1 ? j : outer;
                const size_t off = base + j * lstride + w;
                V v = S1 != 0 ? tile[e] : mkc<V>(T(0), T(0));
                v = op.apply(f, x, y, z0 + w, off, v, pre[k]);
                if (S2 != 0) tile[e] = v;
            }
        }
    }
    pdl_trigger();
    if (S2 != 0) {
        __syncthreads();
        fft_tile<V, S2, E>(tile, st, g.p, g.W, g.fW, g.W, 1);
        for (int e = threadIdx.x; e < ne; e += blockDim.x) {
            const int j = fdiv(e, g.fW), w = e - j * g.W;
            dst[base + j * lstride + w] = tile[e];
        }
    }
    op.end(reinterpret_cast<double*>(tile), blockIdx.x + (size_t)blockIdx.y * gridDim.x);
}

// ---- launches of the run-time passes ----
// Compiled in line_f32.cu and line_f64.cu (FTSP_LINE_ALL in engine.cuh): the
// radix stages are functions, and a compilation that takes the functions of a
// file one by one (-split-compile) costs these passes up to 1.6 times (bond
// pass at 486 x 64 x 64 complex64 72 us, 117 with it; 243 x 16 x 20 27 and 35).
template <class K>
inline cudaError_t pass_smem(K kernel, size_t bytes)
{
    return bytes > 48 * 1024 ? cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) : cudaSuccess;
}
template <typename T, int E, int S1, int S2, class Op>
cudaError_t plane_launch(const PlaneGeom& g, const cplx<T>* src, cplx<T>* dst, int nf, size_t fstride, const cplx<T>* twy,
                         const cplx<T>* twz, int threads, size_t smem, const Op& op, cudaStream_t stream)
{
    auto k = k_plane<T, E, S1, S2, Op>;
    const cudaError_t e = pass_smem(k, smem);
    if (e != cudaSuccess) return e;
    k<<<dim3(g.m1, nf), threads, smem, stream>>>(g, src, dst, fstride, twy, twz, op);
    return cudaGetLastError();
}
template <typename T, int E, int DIM, int S1, int S2, class Op>
cudaError_t strided_launch(const LineGeom& g, const cplx<T>* src, cplx<T>* dst, int nf, size_t fstride, const cplx<T>* tw,
                           int threads, size_t smem, const Op& op, cudaStream_t stream)
{
    auto k = k_strided<T, E, DIM, S1, S2, Op>;
    const cudaError_t e = pass_smem(k, smem);
    if (e != cudaSuccess) return e;
    k<<<dim3((DIM == 1 ? g.m1 : g.m2) * (g.m3 / g.W), nf), threads, smem, stream>>>(g, src, dst, fstride, tw, op);
    return cudaGetLastError();
}
template <typename T, int E, int S1, int S2, class Op>
cudaError_t zline_launch(const LineGeom& g, const cplx<T>* src, cplx<T>* dst, int nf, size_t fstride, const cplx<T>* tw,
                         int threads, size_t smem, const Op& op, cudaStream_t stream)
{
    auto k = k_zline<T, E, S1, S2, Op>;
    const cudaError_t e = pass_smem(k, smem);
    if (e != cudaSuccess) return e;
    k<<<dim3(g.m1 * g.m2 / g.B, nf), threads, smem, stream>>>(g, src, dst, fstride, tw, op);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Pointwise ops
// ---------------------------------------------------------------------------
// Op interface: begin() once per thread; load(f, g) issues the global loads
// an element needs and returns them (the kernels batch PB elements so that
// many loads are in flight); apply(f, x, y, z, g, v, pre) does the element's
// arithmetic and stores and returns the value for the second transform;
// end(scratch, cta) closes per-block reductions.
template <typename T>
struct OpIdentity {
    struct Pre {};
    __device__ __forceinline__ void begin() {}
    __device__ __forceinline__ Pre load(int, size_t) const { return Pre{}; }
    __device__ __forceinline__ cplx<T> apply(int, int, int, int, size_t, cplx<T> v, const Pre&) const { return v; }
    __device__ __forceinline__ void end(double*, size_t) {}
};

// Power-of-two renormalisation of the propagators (all optional: a null eF
// turns it off).  Each real-space segment pass records, per CTA, the largest
// component magnitude of the propagator it wrote (pmax_cur), or one maximum
// over the grid (nparts = 0: an atomic maximum into a slot of the segment, which
// the evaluation has zeroed; order-independent); the next pass of
// the same sweep reduces those maxima, scales its output by 2^-d with
// d = floor(log2 max), and accumulates d into a per-segment exponent:
//   qF[s] is stored as qF_true[s] 2^-aF[s],  qB[s] as qB_true[s] 2^-aB[s].
// Scaling by powers of two is exact in binary floating point, so complex128
// results are unchanged while complex64 propagators stay in range.  A density
// or stress contribution of segment s then carries 2^(aF[s] + aB[s+1] - aF[N-1])
// (the partition function is Q_true = mean(qF[N-1]) 2^aF[N-1]).
struct Renorm {
    int* eF;                 // forward exponents aF[0..N) (null: no renormalisation)
    int* eB;                 // backward exponents aB[0..N)
    const float* pmax_prev;  // per-CTA maxima written by the previous pass of this sweep
    float* pmax_cur;         // per-CTA maxima of this pass
    int nparts;              // number of entries of pmax_prev (0: one slot per segment)
    int s;                   // segment index of this pass
    int N;                   // segments of the species
};

__device__ __forceinline__ int max_exponent(float M) { return (M > 0.0f && isfinite(M)) ? ilogbf(M) : 0; }

// the exponent floor(log2 max) of the previous pass's per-CTA maxima; m is
// this thread's share of them (its strided elements), loaded beforehand
__device__ __forceinline__ int reduce_exponent_local(float m)
{
    __shared__ float s_red[32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        float r = 0.0f;
        for (int w = 0; w < (int)((blockDim.x + 31) >> 5); ++w) r = fmaxf(r, s_red[w]);
        s_red[0] = r;
    }
    __syncthreads();
    const float M = s_red[0];
    __syncthreads();
    return max_exponent(M);
}

__device__ __forceinline__ float local_max(const float* pm, int n)
{
    float m = 0.0f;
    for (int i = threadIdx.x; i < n; i += blockDim.x) m = fmaxf(m, pm[i]);
    return m;
}

__device__ __forceinline__ int reduce_exponent(const float* pm, int n) { return reduce_exponent_local(local_max(pm, n)); }

// Chain-propagator pointwise work in the real-space pass of one segment.
// KIND selects the sweep position:
//   forward : q = u * E (u = IFFT of the previous bond, or 1 at s = 0);
//             q is stored as qF[s]; the last segment also sums q for Q.
//   backward: u = exp(+W_s) qB[s] (the previous transform's output, or 1 at
//             s = N-1); phi = qF[s] * u is accumulated into the per-type
//             and charge densities with the species factor (n/V)/Q; the
//             propagation continues with qB[s] = u * E.
enum PropKind { FWD_START = 0, FWD_MID = 1, FWD_LAST = 2, FWD_SINGLE = 3, BWD_START = 4, BWD_MID = 5, BWD_LAST = 6, BWD_SINGLE = 7 };

template <typename T, int KIND>
struct OpProp {
    using V = cplx<T>;
    const V* E;              // exp(-W) of the segment's class
    V* qstore;               // forward: qF[s]
    const V* qread;          // backward: qF[s]
    V* rho_type;             // backward: density accumulator of the segment's type
    V* rho_charge;           // backward: charge accumulator (null when z == 0)
    T z;                     // segment valence
    const double2* factor;   // backward: species factor (n/V)/Q (Q of the stored, scaled qF)
    double2* partial;        // forward last: per-CTA sums of q
    Renorm rn;               // renormalisation (rn.eF null: off)
    bool store_u;            // forward: store u = q / E (renormalised) instead of q
    double acc[2];
    float amax;
    float pm_local;          // this thread's share of the previous maxima (preload)
    bool preloaded;
    T fr, fi;                // density factor (with the segment's exponent folded in)
    T oscale;                // output scale 2^-d

    static constexpr bool FWD = KIND <= FWD_SINGLE;
    static constexpr bool NEED_E = KIND == FWD_START || KIND == FWD_MID || KIND == FWD_LAST || KIND == FWD_SINGLE ||
                                   KIND == BWD_START || KIND == BWD_MID;
    // global loads per point (the forward passes read only the class table)
    static constexpr int LOADS = FWD ? 1 : 4;
    static constexpr bool MAX_OUT = KIND == FWD_START || KIND == FWD_MID || KIND == BWD_START || KIND == BWD_MID;
    struct Pre {
        V e, q, r, c;
    };

    // loads the previous pass's per-CTA maxima early (kernels that call it
    // right after the dependency wait hide the latency behind their first
    // transform stages; begin() reduces them)
    __device__ __forceinline__ void preload()
    {
        preloaded = false;
        if ((KIND == FWD_MID || KIND == FWD_LAST || KIND == BWD_MID) && rn.eF) {
            pm_local = rn.nparts ? local_max(rn.pmax_prev, rn.nparts) : *rn.pmax_prev;
            preloaded = true;
        }
    }
    __device__ __forceinline__ int prev_exponent() const
    {
        if (rn.nparts == 0) return max_exponent(preloaded ? pm_local : *rn.pmax_prev);
        return preloaded ? reduce_exponent_local(pm_local) : reduce_exponent(rn.pmax_prev, rn.nparts);
    }
    __device__ __forceinline__ void begin()
    {
        acc[0] = acc[1] = 0.0;
        amax = 0.0f;
        oscale = T(1);
        int dens_exp = 0;
        if (rn.eF) {
            const bool first = blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0;
            if (KIND == FWD_START || KIND == FWD_SINGLE) {
                if (first) rn.eF[0] = 0;
            } else if (KIND == FWD_MID || KIND == FWD_LAST) {
                const int d = prev_exponent();
                oscale = (T)ldexp(1.0, -d);
                if (first) rn.eF[rn.s] = rn.eF[rn.s - 1] + d;
            } else if (KIND == BWD_START || KIND == BWD_SINGLE) {
                if (first) rn.eB[rn.s] = 0;
            } else if (KIND == BWD_MID) {
                const int d = prev_exponent();
                oscale = (T)ldexp(1.0, -d);
                if (first) rn.eB[rn.s] = rn.eB[rn.s + 1] + d;
                dens_exp = rn.eF[rn.s] + rn.eB[rn.s + 1] - rn.eF[rn.N - 1];
            } else {   // BWD_LAST (s = 0)
                dens_exp = rn.eF[0] + rn.eB[1] - rn.eF[rn.N - 1];
            }
        }
        if (!FWD) {
            const double2 fc = *factor;
            fr = T(ldexp(fc.x, dens_exp));
            fi = T(ldexp(fc.y, dens_exp));
        }
    }
    __device__ __forceinline__ Pre load(int, size_t g) const
    {
        Pre p;
        if (NEED_E) p.e = E[g];
        if (!FWD) {
            p.q = qread[g];
            p.r = rho_type[g];
            if (rho_charge) p.c = rho_charge[g];
        }
        return p;
    }
    __device__ __forceinline__ void track(V q)
    {
        if (MAX_OUT) amax = fmaxf(amax, fmaxf(fabsf((float)q.x), fabsf((float)q.y)));
    }
    __device__ __forceinline__ V apply(int, int, int, int, size_t g, V u, const Pre& p)
    {
        if (FWD) {
            V q = (KIND == FWD_START || KIND == FWD_SINGLE) ? p.e : cmul(u, p.e);
            if (KIND == FWD_MID || KIND == FWD_LAST) q = cscale(q, oscale);
            if (store_u) {
                if (KIND == FWD_MID || KIND == FWD_LAST) qstore[g] = cscale(u, oscale);
            } else {
                qstore[g] = q;
            }
            track(q);
            if (KIND == FWD_LAST || KIND == FWD_SINGLE) {
                acc[0] += (double)q.x;
                acc[1] += (double)q.y;
            }
            return q;
        } else {
            const V phi = (KIND == BWD_START || KIND == BWD_SINGLE) ? p.q : cmul(p.q, u);
            const V w = cmul(phi, mkc<V>(fr, fi));
            rho_type[g] = cadd(p.r, w);
            if (rho_charge) rho_charge[g] = cadd(p.c, cscale(w, z));
            if (KIND == BWD_START) {
                track(p.e);
                return p.e;
            }
            if (KIND == BWD_MID) {
                const V q = cscale(cmul(u, p.e), oscale);
                track(q);
                return q;
            }
            return u;
        }
    }
    __device__ __forceinline__ void end(double* scratch, size_t cta)
    {
        if (KIND == FWD_LAST || KIND == FWD_SINGLE) {
            __syncthreads();
            block_sum<2>(acc, scratch);
            if (threadIdx.x == 0) partial[cta] = make_double2(acc[0], acc[1]);
        }
        if (MAX_OUT && rn.eF) {
            __syncthreads();
            float* sm = reinterpret_cast<float*>(scratch);
            float m = amax;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
            if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = m;
            __syncthreads();
            if (threadIdx.x == 0) {
                float r = 0.0f;
                for (int w = 0; w < (int)((blockDim.x + 31) >> 5); ++w) r = fmaxf(r, sm[w]);
                // non-negative floats order like their bits
                if (rn.nparts == 0) atomicMax(reinterpret_cast<int*>(rn.pmax_cur), __float_as_int(r));
                else rn.pmax_cur[cta] = r;
            }
        }
    }
};

// Bond pointwise work in the k-space (x) pass of one bond s -> s+1.
//   forward : F = DFT(qF[s]) (sign -1); optionally stored for the stress;
//             output F * Phi_s / V.
//   backward: B' = DFT_{+}(qB[s+1]) (sign +1, i.e. B(-k)); optionally the
//             connectivity stress sums  sum_k k_a k_b Phi_s F_s B'  (weighted
//             by b_s^2 and the species factor) are accumulated; output
//             B' * Phi_s / V.
// Phi_s(k) = exp(-b^2 k^2/6) is separable: phix[kx] phiy[ky] phiz[kz].
template <typename T, bool FWD, bool STRESS>
struct OpBond {
    using V = cplx<T>;
    V* Fstore;
    const V* Fread;
    const T* phix;
    const T* phiy;
    const T* phiz;
    const double* kx;
    const double* ky;
    const double* kz;
    T invV;
    double b2;
    const double2* factor;
    double2* partial;        // [cta][6] accumulated across bonds
    const int* eF;           // renormalisation exponents (null: off)
    const int* eB;
    int s, N;                // bond s -> s+1 of a species with N segments
    double acc[12];
    static constexpr int LOADS = STRESS ? 4 : 0;   // global loads per point (the stress sums need the registers of four)
    struct Pre {
        V F;
    };

    __device__ __forceinline__ void begin()
    {
        if (STRESS) {
#pragma unroll
            for (int c = 0; c < 12; ++c) acc[c] = 0.0;
        }
    }
    __device__ __forceinline__ Pre load(int, size_t g) const
    {
        Pre p;
        if (!FWD && STRESS) p.F = Fread[g];
        return p;
    }
    // For kernels that stage the x factors themselves (x_value, in shared
    // memory): column() gives the factor of a thread's column, once, and
    // apply_x() is apply() with the x factor and the column factor given.
    using XVal = T;
    using Column = T;
    __device__ __forceinline__ T x_value(int x) const { return phix[x]; }
    __device__ __forceinline__ T column(int, int y, int z) const { return __ldg(phiy + y) * __ldg(phiz + z); }
    __device__ __forceinline__ V apply(int f, int x, int y, int z, size_t g, V v, const Pre& pre)
    {
        // read-only loads: they do not alias the Fstore writes, so the y and z
        // factors (fixed for a thread's column) are loaded once
        return apply_x(f, x, y, z, g, v, pre, __ldg(phix + x), column(f, y, z));
    }
    __device__ __forceinline__ V apply_x(int, int x, int y, int z, size_t g, V v, const Pre& pre, T px, T pyz)
    {
        const T phi = px * pyz;
        if (FWD) {
            if (Fstore) Fstore[g] = v;
        } else if (STRESS) {
            const V F = pre.F;
            const V p = cmul(F, v);
            const double pr = (double)p.x * (double)phi, pi = (double)p.y * (double)phi;
            const double ax = kx[x], ay = ky[y], az = kz[z];
            const double kk[6] = {ax * ax, ay * ay, az * az, ax * ay, ax * az, ay * az};
#pragma unroll
            for (int c = 0; c < 6; ++c) {
                acc[2 * c] += kk[c] * pr;
                acc[2 * c + 1] += kk[c] * pi;
            }
        }
        return cscale(v, phi * invV);
    }
    __device__ __forceinline__ void end(double* scratch, size_t cta)
    {
        if (STRESS) {
            __syncthreads();
            block_sum<12>(acc, scratch);
            if (threadIdx.x == 0) {
                const double2 fc = *factor;
                const double w = eF ? ldexp(b2, eF[s] + eB[s + 1] - eF[N - 1]) : b2;
#pragma unroll
                for (int c = 0; c < 6; ++c) {
                    const double sr = w * acc[2 * c], si = w * acc[2 * c + 1];
                    double2 o = partial[cta * 6 + c];
                    o.x += sr * fc.x - si * fc.y;
                    o.y += sr * fc.y + si * fc.x;
                    partial[cta * 6 + c] = o;
                }
            }
        }
    }
};

}  // namespace ftsp

namespace ftsp {


// Source field of output field f of a k-space pass: Op::NSRC entries of
// Op::src where the op declares them (an output computed from another
// field's transform), else f.  The entries are read with constant indices.
template <class Op, class = void>
struct op_has_src : std::false_type {};
template <class Op>
struct op_has_src<Op, std::void_t<decltype(Op::NSRC)>> : std::true_type {};
template <class Op>
__device__ __forceinline__ int op_src_field(const Op& op, int f)
{
    if constexpr (op_has_src<Op>::value) {
        int s = f;
#pragma unroll
        for (int k = 0; k < Op::NSRC; ++k)
            if (k == f) s = op.src[k];
        return s;
    } else {
        return f;
    }
}

// Global loads per point of a pointwise op (Op::LOADS where declared, else 4).
template <class Op, class = void>
struct op_loads {
    static constexpr int value = 4;
};
template <class Op>
struct op_loads<Op, std::void_t<decltype(Op::LOADS)>> {
    static constexpr int value = Op::LOADS;
};

// ops with x_value(), column() and apply_x()
template <class Op, class = void>
struct op_has_xtab : std::false_type {};
template <class Op>
struct op_has_xtab<Op, std::void_t<typename Op::XVal>> : std::true_type {};
template <class Op, bool = op_has_xtab<Op>::value>
struct op_xval {
    using type = char;
    using column = char;
};
template <class Op>
struct op_xval<Op, true> {
    using type = typename Op::XVal;
    using column = typename Op::Column;
};

// op.preload() where the op declares it
template <class Op>
__device__ __forceinline__ auto op_preload_if(Op& op, int) -> decltype(op.preload(), void()) { op.preload(); }
template <class Op>
__device__ __forceinline__ void op_preload_if(Op&, long) {}
template <class Op>
__device__ __forceinline__ void op_preload(Op& op) { op_preload_if(op, 0); }

}  // namespace ftsp
