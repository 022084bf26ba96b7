// EXACT-precision kernels of libdcn for problems large enough to pay for a layout pass: sampling, contraction and
// scatter on the CUDA cores in the tensor dtype (fp32 or fp64), over a channels-last copy of the input.
//
// The kernels of dcn_simt.cu read and scatter the caller's NC(L)HW planes one 4-byte value at a time, locate the
// sampling point again for every channel, and are bound by that: 8.3 ms for a step of 48 GFLOP (config 4, fp32), 9 %
// of the FFMA rate.  Here one pass in front (exact_prep_kernel, a single launch) makes
//   xcl [N][in volume][C4]      channels-last copy; channels padded to whole vectors per segment (see ExactGeom)
//   pts [dg][kv][N * ov]        every sampling point located once: low corner, coinciding-corner bits, fractions
//   w2  [G][K'][Og4]            (forward)  weight in GEMM-K order k' = tap * Cg4 + channel, output channels fastest
//   wt  [G][Og][K']             (backward) weight in the same order, k' fastest
// so that one corner costs one 16-byte load (or one 16-byte reduction) per four channels, and three FFMA kernels with
// 16-deep double-buffered operand tiles do the rest:
//   exact_forward_kernel   y[o, P]      = sum_k' w2[k', o] * sample(k', P), parts of the K range where tiles alone leave SMs
//                                         idle, added in part order by the last of a tile to finish: reproducible
//   exact_data_kernel      col[k', P]   = sum_o  wt[o, k'] * dy[o, P], consumed from registers: reductions into a
//                                         channels-last dX, corner dot products for dOffset
//   exact_weight_kernel    dW[o, k']    = sum_P  dy[o, P] * sample(k', P), position range split over CTAs, one slice of
//                                         a scratch each (summed in slice order: reproducible)
// Arithmetic is that of dcn_simt.cu: fp32 / fp64 throughout, the same point rule and interpolation order.
// Replaces deform3d/lib/deform_conv3d_cuda.cpp:90-336 with the kernels of deform3d/lib/deform_conv3d_cuda_kernel.cu:
// 62-131, 175-298, 340-485 (and the 2-D / plain twins) like dcn_simt.cu does.
#include <type_traits>

#include "dcn_internal.h"

namespace dcn {

namespace {

constexpr int kXThreads = 256;
constexpr int kBK = 16;              // depth of one operand tile
constexpr int kPtsPerThread = 4;

// Channels of one convolution group that share a deformable group are a segment: S consecutive channels, stored as S4
// (a whole number of vectors; the pad channels are zero).  Uniform because one of Cg, cpg divides the other.
struct ExactGeom {
    int S, S4, segs;                 // segs: segments per convolution group
    int Cg4, C4;                     // padded channels per convolution group / in all
    int Kp, Kp16, Kp64;              // kv * Cg4, and rounded up to the tile depths
    int Og4;
    int split;                       // a deformable group spans several convolution groups
    FastDiv d_Cg4, d_S4, d_Og4, d_Kp64;
};

template <typename T, int V>
struct Vec {
    T v[V];
};

template <typename T, int V>
__device__ __forceinline__ Vec<T, V> load_vec(const T* p) {
    Vec<T, V> r;
    if constexpr (V * sizeof(T) == 16) {
        const uint4 q = gload(reinterpret_cast<const uint4*>(p));
        memcpy(&r, &q, 16);
    } else {
#pragma unroll
        for (int i = 0; i < V; ++i) r.v[i] = gload(p + i);
    }
    return r;
}

template <typename T, int V>
__device__ __forceinline__ void add_vec(T* p, const T (&v)[V]) {
    if constexpr (std::is_same<T, float>::value && V == 4) {
        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]));
    } else {
#pragma unroll
        for (int i = 0; i < V; ++i) atomicAdd(p + i, v[i]);
    }
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool ok) {
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
    const int n = ok ? 16 : 0;       // 0: the sixteen bytes become zero
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// ---- sampling points ---------------------------------------------------------------------------------------------
// One entry per (deformable group, tap, position).  bits: low-corner index (28 bits) | hi != lo on axis w, h, l (bits
// 28..30) | invalid (bit 31; then bits 2a, 2a+1 say whether axis a lies below or beyond the out-of-bounds thresholds).
template <typename T> struct Entry;
template <> struct __align__(16) Entry<float> { uint32_t bits; float l[3]; };
template <> struct __align__(16) Entry<double> { uint32_t bits; uint32_t pad; double l[3]; };

template <typename T, int D>
__device__ __forceinline__ Entry<T> make_entry(const Geom& g, const Pt<T, D>& s) {
    Entry<T> e;
    e.l[0] = e.l[1] = e.l[2] = (T)0;
    if (s.valid) {
        int idx[1 << D];
        corner_indices<T, D>(g, s, idx);
        e.bits = (uint32_t)idx[0];
#pragma unroll
        for (int a = 0; a < D; ++a) {
            if (s.hi[a] != s.lo[a]) e.bits |= 1u << (28 + (D - 1 - a));
            e.l[a] = s.lw[a];
        }
    } else {
        e.bits = 1u << 31;
#pragma unroll
        for (int a = 0; a < D; ++a) {
            const T t = oob_term<T>(g, s.p[a], (T)1);
            if (t < (T)0) e.bits |= 1u << (2 * a);
            if (t > (T)0) e.bits |= 2u << (2 * a);
        }
    }
    return e;
}

template <typename T>
__device__ __forceinline__ Entry<T> load_entry(const Entry<T>* p) {
    Entry<T> e;
    const uint4* q = reinterpret_cast<const uint4*>(p);
    uint4 t[sizeof(Entry<T>) / 16];
#pragma unroll
    for (int i = 0; i < (int)(sizeof(Entry<T>) / 16); ++i) t[i] = gload(q + i);
    memcpy(&e, t, sizeof(e));
    return e;
}

// element offsets of the 2^D corners in a channels-last sample, relative to the channel
template <int D>
__device__ __forceinline__ void entry_corners(const Geom& g, const ExactGeom& xg, uint32_t bits, uint32_t (&at)[1 << D]) {
    const uint32_t c4 = (uint32_t)xg.C4;
    const uint32_t base = (bits & 0x0fffffffu) * c4;
    const uint32_t sw = (bits & (1u << 28)) ? c4 : 0u;
    const uint32_t sh = (bits & (1u << 29)) ? c4 * (uint32_t)g.in[2] : 0u;
    const uint32_t sl = (D == 3 && (bits & (1u << 30))) ? c4 * (uint32_t)(g.in[1] * g.in[2]) : 0u;
#pragma unroll
    for (int e = 0; e < (1 << D); ++e) at[e] = base + ((e & 1) ? sw : 0u) + ((e & 2) ? sh : 0u) + ((e & 4) ? sl : 0u);
}

template <typename T, int D>
__device__ __forceinline__ void entry_weights(const Entry<T>& e, Pt<T, D>& s) {
#pragma unroll
    for (int a = 0; a < D; ++a) {
        s.lw[a] = e.l[a];
        s.hw[a] = (T)1 - e.l[a];
    }
}

// deformable group of channel c4 (padded, within convolution group j)
__device__ __forceinline__ int group_of(const Geom& g, const ExactGeom& xg, int j, uint32_t c4) {
    return xg.split ? (int)g.d_cpg.div((uint32_t)(j * g.Cg)) : j * xg.segs + (int)xg.d_S4.div(c4);
}

// ---- vectors of V channels: fp32 works on packed pairs (one instruction slot, each lane an IEEE operation) ------------
__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// Lanes of a vector: V values, or V / 2 packed pairs in fp32.
template <typename T, int V>
struct Lanes {
    static constexpr int N = V;
    using L = T;
    static __device__ __forceinline__ L same(T a) { return a; }
    static __device__ __forceinline__ L mul(L a, L b) { return a * b; }
    static __device__ __forceinline__ L fma(L a, L b, L c) { return a * b + c; }
    static __device__ __forceinline__ void load(const T (&v)[V], L (&l)[N]) {
#pragma unroll
        for (int i = 0; i < N; ++i) l[i] = v[i];
    }
    static __device__ __forceinline__ void store(const L (&l)[N], T (&v)[V]) {
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = l[i];
    }
    static __device__ __forceinline__ T sum(const L (&l)[N]) {
        T r = l[0];
#pragma unroll
        for (int i = 1; i < N; ++i) r += l[i];
        return r;
    }
};
template <>
struct Lanes<float, 4> {
    static constexpr int N = 2;
    using L = uint64_t;
    static __device__ __forceinline__ L same(float a) { return pack2(a, a); }
    static __device__ __forceinline__ L mul(L a, L b) { return mul2(a, b); }
    static __device__ __forceinline__ L fma(L a, L b, L c) { return fma2(a, b, c); }
    static __device__ __forceinline__ void load(const float (&v)[4], L (&l)[2]) {
        l[0] = pack2(v[0], v[1]);
        l[1] = pack2(v[2], v[3]);
    }
    static __device__ __forceinline__ void store(const L (&l)[2], float (&v)[4]) {
        unpack2(l[0], v[0], v[1]);
        unpack2(l[1], v[2], v[3]);
    }
    static __device__ __forceinline__ float sum(const L (&l)[2]) {
        float a, b, c, d;
        unpack2(l[0], a, b);
        unpack2(l[1], c, d);
        return (a + b) + (c + d);
    }
};

// Interpolation of V channels in the reference's order (along w, then h, then l), like interp().
template <typename T, int D, int V>
__device__ __forceinline__ void interp_vec(const Pt<T, D>& s, const Vec<T, V> (&cv)[1 << D], T (&out)[V]) {
    using Ln = Lanes<T, V>;
    typename Ln::L c[1 << D][Ln::N];
#pragma unroll
    for (int e = 0; e < (1 << D); ++e) Ln::load(cv[e].v, c[e]);
#pragma unroll
    for (int a = D - 1; a >= 0; --a) {                                 // halve the corners along axis a
        const auto hw = Ln::same(s.hw[a]), lw = Ln::same(s.lw[a]);
        const int n = 1 << a;
#pragma unroll
        for (int e = 0; e < n; ++e)
#pragma unroll
            for (int i = 0; i < Ln::N; ++i) c[e][i] = Ln::fma(c[2 * e + 1][i], lw, Ln::mul(c[2 * e][i], hw));
    }
    Ln::store(c[0], out);
}

// N consecutive values from shared memory, in the widest loads that N allows
template <typename T, int N>
__device__ __forceinline__ void load_row(const T* p, T (&r)[N]) {
    constexpr int B = N * (int)sizeof(T);
    if constexpr (B % 16 == 0) {
#pragma unroll
        for (int i = 0; i < B / 16; ++i) {
            const uint4 q = reinterpret_cast<const uint4*>(p)[i];
            memcpy(reinterpret_cast<char*>(r) + 16 * i, &q, 16);
        }
    } else if constexpr (B % 8 == 0) {
#pragma unroll
        for (int i = 0; i < B / 8; ++i) {
            const uint2 q = reinterpret_cast<const uint2*>(p)[i];
            memcpy(reinterpret_cast<char*>(r) + 8 * i, &q, 8);
        }
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) r[i] = p[i];
    }
}

// One item: a vector of V samples of tap / channel run (key, c) at one position.  Its corner values travel by cp.async
// into slots of shared memory that only the issuing thread reads, so that kAhead further items can be in flight without
// registers to hold them: with one item in registers the forward and weight kernels waited for corners half of the time
// (config 4: 0.80 and 0.73 ms, FMA pipe 40 % busy).
// 3-D fp32 keeps one item ahead, not two: eight corners an item, and at three CTAs per SM the third stage would push the
// shared-memory carve-out from 196 to 228 KB and leave 28 KB of L1 instead of 60 (config 4: forward 0.69 -> 0.65, weight
// 0.68 -> 0.64 ms; 2-D is 1 % slower with one).
template <typename T, int D, bool DEFORM>
constexpr int kAheadOf = sizeof(T) == 4 && D == 3 && DEFORM ? 1 : 2;

template <int BYTES>
__device__ __forceinline__ void cp_async_small(void* smem, const void* gmem, bool ok) {
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
    const int n = ok ? BYTES : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(s), "l"(gmem), "n"(BYTES), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait_group() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <typename T, int D, bool DEFORM, int V, int NT>
struct Sampler {
    static constexpr int kAhead = kAheadOf<T, D, DEFORM>, kStages = kAhead + 1;
    static constexpr int NC = DEFORM ? (1 << D) : 1, VB = V * (int)sizeof(T);
    static constexpr int kBytes = kStages * NC * NT * VB;
    char* slots;                     // [stage][corner][thread]
    Entry<T> e[kStages];             // of the items in flight, the one to finish next first (deformable only)

    __device__ __forceinline__ char* slot(int stage, int corner) const { return slots + ((stage * NC + corner) * NT) * VB; }

    // xn: the sample's block of xcl plus the channel; idx < 0: nothing to read (plain convolution)
    __device__ __forceinline__ void issue(const Geom& g, const ExactGeom& xg, int stage, const T* xn, const Entry<T>& entry,
                                          bool ok, int idx) {
        if constexpr (DEFORM) {
            Entry<T>& mine = e[kAhead];
            mine = entry;
            if (!ok) mine.bits = 1u << 31;
            if (!(mine.bits >> 31)) {
                uint32_t at[1 << D];
                entry_corners<D>(g, xg, entry.bits, at);
#pragma unroll
                for (int i = 0; i < (1 << D); ++i) cp_async_small<VB>(slot(stage, i), xn + at[i], true);
            }
        } else {
            const bool read = ok && idx >= 0;
            cp_async_small<VB>(slot(stage, 0), read ? xn + (uint32_t)idx * (uint32_t)xg.C4 : xn, read);
        }
    }
    // before each issue: the entries move up
    __device__ __forceinline__ void advance() {
        if constexpr (DEFORM) {
#pragma unroll
            for (int i = 0; i < kAhead; ++i) e[i] = e[i + 1];
        }
    }
    // the values of the oldest item in flight (its copies have arrived)
    __device__ __forceinline__ Vec<T, V> finish(int stage) {
        Vec<T, V> r;
        if constexpr (DEFORM) {
            if (e[0].bits >> 31) {
#pragma unroll
                for (int v = 0; v < V; ++v) r.v[v] = (T)0;
            } else {
                Vec<T, V> cv[1 << D];
#pragma unroll
                for (int i = 0; i < (1 << D); ++i) load_row<T, V>(reinterpret_cast<const T*>(slot(stage, i)), cv[i].v);
                Pt<T, D> s;
                entry_weights<T, D>(e[0], s);
                interp_vec<T, D, V>(s, cv, r.v);
            }
        } else {
            load_row<T, V>(reinterpret_cast<const T*>(slot(stage, 0)), r.v);
        }
        return r;
    }
};

// Place of a thread in the 16 x 16 grid of register tiles: a warp covers 8 x 4 of it, so that both operand reads of a
// step (16 bytes per lane) are one 128-byte wavefront each (16 x 2 took three; shared memory is what these kernels and
// their corner loads queue for: L1 at 70 % of its rate in a step of config 4).
__device__ __forceinline__ int tile_x(int tid) { return (tid / 32) % 2 * 8 + tid % 8; }
__device__ __forceinline__ int tile_y(int tid) { return tid / 64 * 4 + tid % 32 / 8; }

// ---- register tiles ----------------------------------------------------------------------------------------------
// acc[R][C] += a[R] x b[C]; fp32 as packed pairs along R (fma.rn.f32x2: two IEEE FMAs in one instruction slot)
template <typename T, int R, int C>
struct Acc {
    T v[R][C];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
            for (int q = 0; q < C; ++q) v[i][q] = (T)0;
    }
    __device__ __forceinline__ void fma(const T (&a)[R], const T (&b)[C]) {
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
            for (int q = 0; q < C; ++q) v[i][q] += a[i] * b[q];
    }
    __device__ __forceinline__ T at(int i, int q) const { return v[i][q]; }
    __device__ __forceinline__ void add(int i, int q, T a) { v[i][q] += a; }
};
template <int R, int C>
struct Acc<float, R, C> {
    static_assert(R % 2 == 0, "pairs along R");
    uint64_t v[R / 2][C];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int i = 0; i < R / 2; ++i)
#pragma unroll
            for (int q = 0; q < C; ++q) v[i][q] = 0ull;
    }
    __device__ __forceinline__ void fma(const float (&a)[R], const float (&b)[C]) {
        uint64_t ap[R / 2], bp[C];
#pragma unroll
        for (int i = 0; i < R / 2; ++i) asm("mov.b64 %0, {%1, %2};" : "=l"(ap[i]) : "f"(a[2 * i]), "f"(a[2 * i + 1]));
#pragma unroll
        for (int q = 0; q < C; ++q) asm("mov.b64 %0, {%1, %1};" : "=l"(bp[q]) : "f"(b[q]));
#pragma unroll
        for (int i = 0; i < R / 2; ++i)
#pragma unroll
            for (int q = 0; q < C; ++q) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(v[i][q]) : "l"(ap[i]), "l"(bp[q]));
    }
    __device__ __forceinline__ float at(int i, int q) const {
        float lo, hi;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v[i / 2][q]));
        return (i & 1) ? hi : lo;
    }
    __device__ __forceinline__ void add(int i, int q, float a) {
        float lo, hi;
        unpack2(v[i / 2][q], lo, hi);
        v[i / 2][q] = (i & 1) ? pack2(lo, hi + a) : pack2(lo + a, hi);
    }
};

// ------------------------------------------------------------------------------------------------------------------
// Prologue of a pass, one launch: block ranges for the bias gradient, the input copy, the points, the weight and a zero fill.
// ------------------------------------------------------------------------------------------------------------------
template <typename T>
constexpr int kCopyTile = sizeof(T) == 4 ? 64 : 32;      // side of a transpose tile

template <typename T>
struct PrepArgs {
    const T *x, *off, *w, *dy;
    T *xcl, *wk, *zero, *zero2, *dbias;      // wk: w2 (forward) or wt (backward); zero: dX scratch, or the tiles' counters
    Entry<T>* pts;
    size_t zero_n, zero2_n;          // elements
    unsigned nb, nx, np, nw, nz;     // blocks of each part
    unsigned tx, ty;                 // input copy: tiles along the positions / channels
    unsigned bpk;                    // points: blocks of one (deformable group, tap)
    int backward;
};

template <typename T, int D>
__global__ void __launch_bounds__(kXThreads)
exact_prep_kernel(const Geom g, const ExactGeom xg, const PrepArgs<T> a) {
    constexpr int TC = kCopyTile<T>;
    __shared__ T tile[TC][TC + 1];
    pdl_trigger();
    pdl_wait();
    unsigned b = blockIdx.x;
    if (b < a.nb) {                                                    // bias gradient: one output channel
        T s = (T)0;
        for (long long i = threadIdx.x; i < g.P; i += kXThreads) {
            uint32_t n, opos;
            g.d_ov.divmod((uint32_t)i, n, opos);
            s += gload(a.dy + ((size_t)n * g.O + b) * g.ov + opos);
        }
        T* red = &tile[0][0];
        red[threadIdx.x] = s;
        __syncthreads();
        for (int st = kXThreads / 2; st > 0; st >>= 1) {
            if ((int)threadIdx.x < st) red[threadIdx.x] += red[threadIdx.x + st];
            __syncthreads();
        }
        if (threadIdx.x == 0) a.dbias[b] = red[0];
        return;
    }
    b -= a.nb;
    if (b < a.nx) {                                                    // x -> xcl, TC channels x TC positions
        const unsigned px = b % a.tx, r = b / a.tx, cy = r % a.ty, n = r / a.ty;
        const int tx = threadIdx.x % 32, ty = threadIdx.x / 32;
        const int p0 = (int)px * TC, c0 = (int)cy * TC;
        const T* xn = a.x + (size_t)n * g.C * g.iv;
        T v[TC / 8][TC / 32];                                          // all loads in flight together
#pragma unroll
        for (int i = 0; i < TC / 8; ++i) {
            const int c4 = c0 + ty + i * 8;
            uint32_t seg, r4;
            xg.d_S4.divmod((uint32_t)c4, seg, r4);
            const bool ok = c4 < xg.C4 && (int)r4 < xg.S;
            const T* xc = xn + (size_t)(ok ? seg * xg.S + r4 : 0) * g.iv;
#pragma unroll
            for (int h = 0; h < TC / 32; ++h) {
                const int p = p0 + h * 32 + tx;
                v[i][h] = ok && p < g.iv ? gload(xc + p) : (T)0;
            }
        }
#pragma unroll
        for (int i = 0; i < TC / 8; ++i)
#pragma unroll
            for (int h = 0; h < TC / 32; ++h) tile[ty + i * 8][h * 32 + tx] = v[i][h];
        __syncthreads();
        T* on = a.xcl + (size_t)n * g.iv * xg.C4;
#pragma unroll
        for (int i = 0; i < TC / 8; ++i) {
            const int p = p0 + ty + i * 8;
#pragma unroll
            for (int h = 0; h < TC / 32; ++h) {
                const int c4 = c0 + h * 32 + tx;
                if (p < g.iv && c4 < xg.C4) on[(size_t)p * xg.C4 + c4] = tile[h * 32 + tx][ty + i * 8];
            }
        }
        return;
    }
    b -= a.nx;
    if (b < a.np) {                                                    // sampling points
        const unsigned key = b / a.bpk;
        uint32_t grp, tap;
        g.d_kv.divmod(key, grp, tap);
        const long long P0 = (long long)(b - key * a.bpk) * (kPtsPerThread * kXThreads) + threadIdx.x;
        T offv[kPtsPerThread][D];
        OutPos op[kPtsPerThread];
#pragma unroll
        for (int i = 0; i < kPtsPerThread; ++i) {                      // all offset loads in flight together
            const long long P = P0 + i * kXThreads;
            op[i] = decompose_pos(g, P < g.P ? P : 0);
            const T* ob = offset_ptr<T, D>(g, offset_block<T, D>(g, a.off, op[i].n), (int)grp, (int)tap, op[i]);
#pragma unroll
            for (int d = 0; d < D; ++d) offv[i][d] = gload(ob + (size_t)d * g.ov);
        }
#pragma unroll
        for (int i = 0; i < kPtsPerThread; ++i) {
            const long long P = P0 + i * kXThreads;
            if (P >= g.P) break;
            Pt<T, D> s;
            locate_with<T, D>(g, offv[i], (int)tap, op[i], s);
            a.pts[(size_t)key * (size_t)g.P + (size_t)P] = make_entry<T, D>(g, s);
        }
        return;
    }
    b -= a.np;
    if (b < a.nw) {                                                    // weight, reordered and padded with zeros
        const size_t rows = a.backward ? (size_t)g.Og : (size_t)xg.Kp16, cols = a.backward ? xg.Kp64 : xg.Og4;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const size_t e = ((size_t)b * 4 + i) * kXThreads + threadIdx.x;
            if (e >= rows * cols * g.G) return;
            uint32_t row, col;
            (a.backward ? xg.d_Kp64 : xg.d_Og4).divmod((uint32_t)e, row, col);
            const uint32_t j = row / (uint32_t)rows;
            row -= j * (uint32_t)rows;
            const uint32_t kp = a.backward ? col : row, o = a.backward ? row : col;
            T v = (T)0;
            if ((int)kp < xg.Kp && (int)o < g.Og) {
                uint32_t tap, c4, seg, r4;
                xg.d_Cg4.divmod(kp, tap, c4);
                xg.d_S4.divmod(c4, seg, r4);
                if ((int)r4 < xg.S) v = gload(a.w + ((size_t)(j * g.Og + o) * g.Cg + seg * xg.S + r4) * g.kv + tap);
            }
            a.wk[e] = v;
        }
        return;
    }
    b -= a.nw;
    constexpr int W = 16 / (int)sizeof(T);                             // dX scratch, or counters; dOffset
    const bool second = b >= a.nz;
    T* z = second ? a.zero2 : a.zero;
    const size_t len = second ? a.zero2_n : a.zero_n;
    if (second) b -= a.nz;
    const size_t whole = (reinterpret_cast<uintptr_t>(z) & 15) == 0 ? len / W : 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const size_t e = ((size_t)b * 4 + i) * kXThreads + threadIdx.x;
        if (e < whole) {
            reinterpret_cast<uint4*>(z)[e] = make_uint4(0u, 0u, 0u, 0u);
        } else {
#pragma unroll
            for (int k = 0; k < W; ++k)
                if (e * W + k < len) z[e * W + k] = (T)0;
        }
    }
}

// ------------------------------------------------------------------------------------------------------------------
// Forward and backward weight: 16 x TY threads of TM x TN outputs each.
// Wide tiles (fp32): 8 x 8 outputs per thread, TY the height (8 * TY output channels).  A step of 16-byte shared loads
// then returns 16 lane-registers for 64 FMAs; the return path (128 bytes a clock) held 4 x 4 and 6 x 4 outputs at half
// of the FMA rate.  Narrow tiles (problems whose wide tiles leave SMs idle; fp64, which runs at half the FMA rate): 64
// columns, 2 x 4 or 4 x 4 outputs, 256 threads, so that a chunk is one item per thread and the chain of a CTA is short.
// The items (vectors of one position) of the next chunk are spread over the FMA steps of this one: copies of the item
// kAhead further on issued, a share of the FMAs, the oldest item interpolated and stored.  Point entries are loaded one
// item before they are needed.  Config 4: forward 2.49 -> 0.69 ms, weight 1.77 -> 0.68 ms against dcn_simt.cu.
// ------------------------------------------------------------------------------------------------------------------
template <typename T, int TN, int TY>
constexpr int kCtasPerSm = sizeof(T) == 8 ? 1 : (TN == 4 ? 2 : (TY == 4 ? 5 : (TY == 8 ? 3 : (TY == 12 ? 2 : 1))));

// first column of the h-th run of four of a thread's TN columns (runs 64 apart, so that the lanes of a warp read
// consecutive 16-byte words)
__device__ __forceinline__ int tile_col(int tx, int h) { return h * 64 + tx * 4; }

// Bs columns are permuted by row in the forward kernel, so that the stores of a warp (a few positions, consecutive rows)
// spread over the banks while the reads stay 16-byte vectors.
template <int V>
__device__ __forceinline__ int bs_perm(int row) { return V == 4 ? (row / 4) % 4 * 8 : (row % 8) * 4; }

template <typename T, int TM, int TN>
__device__ __forceinline__ void tile_step(Acc<T, TM, TN>& acc, const T* arow, const T* brow, int tx, int ty, int perm) {
    T a[TM], b[TN];
    load_row<T, TM>(arow + ty * TM, a);
#pragma unroll
    for (int h = 0; h < TN / 4; ++h) {
        T t[4];
        load_row<T, 4>(brow + (tile_col(tx, h) ^ perm), t);
#pragma unroll
        for (int i = 0; i < 4; ++i) b[4 * h + i] = t[i];
    }
    acc.fma(a, b);
}

// Parts of the K range (grid.z > 1): each stores its sums in a slice of its own, and the CTA that finishes a tile last --
// `done` counts them; nobody waits -- adds the slices in part order and stores y.  Every output is thus written once and
// has one order of summation; reductions into a zeroed y gave the last bits to whichever part came first.
// A thread reads back what the same thread of the other parts stored, 16 bytes per lane and slice vector.  Costs 1.5 us of
// a step against the reductions (6 x 96 -> 96 channels 33x45, four parts: 187.5 -> 189.0 us; plain 8 x 64 -> 128, 56x56
// stride 2, three parts: 99.6 -> 101.3): a tile's slices pass through the one SM that finishes it.
template <typename T, int TM, int TN, int NT>
__device__ __forceinline__ bool fold_parts(Acc<T, TM, TN>& acc, T* slices, unsigned* done, char* smem) {
    constexpr int W = 16 / (int)sizeof(T), E = TM * TN / W;            // 16-byte vectors of a thread
    static_assert(TN % W == 0, "a vector lies within one row of the register tile");
    const int tid = threadIdx.x;
    const size_t tile = (size_t)blockIdx.y * gridDim.x + blockIdx.x;
    T* all = slices + tile * gridDim.z * (TM * TN * NT) + tid * W;
    T* mine = all + (size_t)blockIdx.z * (TM * TN * NT);
#pragma unroll
    for (int e = 0; e < E; ++e) {
        T t[W];
#pragma unroll
        for (int k = 0; k < W; ++k) t[k] = acc.at(e * W / TN, e * W % TN + k);
        uint4 q;
        memcpy(&q, t, 16);
        __stcg(reinterpret_cast<uint4*>(mine + e * (NT * W)), q);
    }
    __threadfence();                                                   // the slice is visible before it is counted
    __syncthreads();                                                   // (also: the operand tiles are done with)
    if (tid == 0) *reinterpret_cast<unsigned*>(smem) = atomicAdd(done + tile, 1u);
    __syncthreads();
    if (*reinterpret_cast<volatile unsigned*>(smem) + 1 != gridDim.z) return false;
    __threadfence();
    acc.clear();
#pragma unroll 2
    for (unsigned z = 0; z < gridDim.z; ++z, all += TM * TN * NT) {
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const uint4 q = gload_cg(reinterpret_cast<const uint4*>(all + e * (NT * W)));
            T t[W];
            memcpy(t, &q, 16);
#pragma unroll
            for (int k = 0; k < W; ++k) acc.add(e * W / TN, e * W % TN + k, t[k]);
        }
    }
    return true;
}

// grid.x: tiles of 16 * TN positions; grid.y: G * ceil(Og / BM); grid.z: parts of the K range (more than one where the
// tiles alone leave SMs idle).  slices, done: see fold_parts; `done` is zeroed by the prologue.
// SPLIT is a kernel of its own: with the fold's registers in the whole-tile one a step of config 4 took 2495 us, not 2408.
template <typename T, int D, bool DEFORM, int V, int TM, int TN, int TY, bool SPLIT>
__global__ void __launch_bounds__(16 * TY, kCtasPerSm<T, TN, TY>)
exact_forward_kernel(const Geom g, const ExactGeom xg, const T* __restrict__ xcl, const Entry<T>* __restrict__ pts,
                     const T* __restrict__ w2, const T* __restrict__ bias, T* __restrict__ y, int chunks_per_part,
                     T* __restrict__ slices, unsigned* __restrict__ done) {
    constexpr int BM = TM * TY, BN = 16 * TN, NT = 16 * TY;
    constexpr int Q = kBK / V, ALL = BN * Q, ITEMS = (ALL + NT - 1) / NT, L16 = 16 / (int)sizeof(T);
    extern __shared__ __align__(16) char smem_x[];
    T (*As)[kBK][BM] = reinterpret_cast<T (*)[kBK][BM]>(smem_x);
    T (*Bs)[kBK][BN] = reinterpret_cast<T (*)[kBK][BN]>(smem_x + 2 * kBK * BM * sizeof(T));
    const int tid = threadIdx.x, tx = tile_x(tid), ty = tile_y(tid);
    const int mt = (g.Og + BM - 1) / BM;
    const int j = blockIdx.y / mt, o0 = (blockIdx.y % mt) * BM;
    const long long P0 = (long long)blockIdx.x * BN;
    const int q = tid % Q;                                            // (NT is a multiple of Q)
    const T* xj = xcl + j * xg.Cg4;
    const T* wg = w2 + (size_t)j * xg.Kp16 * xg.Og4;

    auto load_a = [&](int ch) {
#pragma unroll
        for (int i = 0; i < (kBK * BM / L16 + NT - 1) / NT; ++i) {
            const int e = tid + i * NT;
            if (kBK * BM / L16 % NT != 0 && e >= kBK * BM / L16) break;
            const int row = e / (BM / L16), m = (e % (BM / L16)) * L16;
            const bool ok = o0 + m < xg.Og4;
            cp_async16(&As[ch & 1][row][m], wg + (size_t)(ch * kBK + row) * xg.Og4 + (ok ? o0 + m : 0), ok);
        }
    };
    // Item it of a chunk: rows q*V .. of the chunk at position column(it).  What depends on the position only is kept for
    // the whole kernel, what depends on the chunk is advanced once per chunk, so that an item costs little but its own
    // loads and arithmetic.
    auto column = [&](int it) { return tid / Q + it * (NT / Q); };
    uint32_t pos_ok = 0;                                              // bit it: the position exists
    size_t xoff[ITEMS];                                               // its sample's block in xcl
    int base[DEFORM ? 1 : ITEMS][3];
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
        const bool ok = (ALL % NT == 0 || column(it) < BN) && P0 + column(it) < g.P;
        if (ok) pos_ok |= 1u << it;
        const OutPos op = decompose_pos(g, ok ? P0 + column(it) : 0);
        xoff[it] = (size_t)op.n * (uint32_t)g.iv * (uint32_t)xg.C4;
        if constexpr (!DEFORM) {
            base[it][0] = op.base[0]; base[it][1] = op.base[1]; base[it][2] = op.base[2];
        }
    }
    struct Chunk {                                                    // this thread's rows of one chunk
        int kp;
        uint32_t tap, c;
        const Entry<T>* pk;                                           // entries of its key, at column(0)
    };
    auto chunk = [&](int ch) {
        Chunk k;
        k.kp = ch * kBK + q * V;
        xg.d_Cg4.divmod((uint32_t)k.kp, k.tap, k.c);
        k.pk = nullptr;
        if constexpr (DEFORM) {
            if (k.kp < xg.Kp) k.pk = pts + (size_t)(group_of(g, xg, j, k.c) * g.kv + (int)k.tap) * (size_t)g.P + (size_t)(P0 + column(0));
        }
        return k;
    };
    constexpr int kAhead = kAheadOf<T, D, DEFORM>, kStages = kAhead + 1;
    Sampler<T, D, DEFORM, V, NT> smp;
    smp.slots = smem_x + 2 * kBK * (BM + BN) * sizeof(T) + tid * V * sizeof(T);
    Entry<T> ent;
    auto fetch = [&](const Chunk& k, int it) {                        // the item's point entry
        if constexpr (DEFORM) {
            if (k.kp < xg.Kp && (pos_ok >> it & 1)) ent = load_entry(k.pk + it * (NT / Q));
        }
    };
    auto issue = [&](int stage, const Chunk& k, int it) {             // its corner copies
        const bool ok = k.kp < xg.Kp && (pos_ok >> it & 1);
        int idx = -1;
        if constexpr (!DEFORM) {
            OutPos op;
            op.base[0] = base[it][0]; op.base[1] = base[it][1]; op.base[2] = base[it][2];
            int at;
            if (ok && locate_plain<D>(g, (int)k.tap, op, at)) idx = at;
        }
        smp.issue(g, xg, stage, xj + xoff[it] + k.c, ent, ok, idx);
    };
    int fs = 0, is = 0;                                               // stages of the next item to finish / to issue
    auto finish = [&](int ch, int it) {                               // its values, into the chunk's tile
        const Vec<T, V> r = smp.finish(fs);
        fs = fs + 1 == kStages ? 0 : fs + 1;
        const int n = column(it);
        if (ALL % NT == 0 || n < BN) {
#pragma unroll
            for (int v = 0; v < V; ++v) Bs[ch & 1][q * V + v][n ^ bs_perm<V>(q * V + v)] = r.v[v];
        }
    };

    Acc<T, TM, TN> acc;
    acc.clear();
    const int ch0 = (int)blockIdx.z * chunks_per_part, all = xg.Kp16 / kBK;
    const int ch1 = ch0 + chunks_per_part < all ? ch0 + chunks_per_part : all;
    // Step s issues item s (chunk ch0 + s / ITEMS, it s % ITEMS) and fetches the entry of item s + 1.
    Chunk ki = chunk(ch0), kf = ki;                                   // chunks of the next issue / fetch
    int ci = ch0, cf = ch0;
    auto step = [&](int it) {                                         // it: s % ITEMS, a compile-time constant
        smp.advance();
        if (ci < ch1) issue(is, ki, it);
        cp_async_commit();                                            // (empty at the end: the waits count groups)
        is = is + 1 == kStages ? 0 : is + 1;
        const int nf = (it + 1) % ITEMS;
        if (nf == 0) {
            ki = kf = chunk(++cf);
            ++ci;
            if constexpr (DEFORM) {
                // the entries two chunks on come from DRAM: bring them to L2 (a row of the tile per thread)
                const Chunk far = chunk(cf + 1);
                if (cf + 1 < ch1 && far.kp < xg.Kp && P0 + tid / Q * ITEMS < g.P)
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(far.pk + (tid / Q * ITEMS - column(0))));
            }
        }
        if (cf < ch1) fetch(kf, nf);
    };
    pdl_wait();
    fetch(kf, 0);
    load_a(ch0);                                                      // (completes with the first item)
#pragma unroll
    for (int i = 0; i < kAhead; ++i) step(i % ITEMS);
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
        step((it + kAhead) % ITEMS);
        cp_async_wait_group<kAhead>();
        finish(ch0, it);
    }
    for (int ch = ch0; ch < ch1; ++ch) {
        __syncthreads();
        const bool more = ch + 1 < ch1;
        if (more) load_a(ch + 1);                                     // in the group of the item issued next
#pragma unroll
        for (int it = 0; it < ITEMS; ++it) {
            step((it + kAhead) % ITEMS);
#pragma unroll
            for (int kk = it * kBK / ITEMS; kk < (it + 1) * kBK / ITEMS; ++kk)
                tile_step<T, TM, TN>(acc, As[ch & 1][kk], Bs[ch & 1][kk], tx, ty, bs_perm<V>(kk));
            // the last wait of a chunk also covers the weight tile
            if (it + 1 < ITEMS) cp_async_wait_group<kAhead>();
            else cp_async_wait_group<(kAhead < ITEMS - 1 ? kAhead : ITEMS - 1)>();
            if (more) finish(ch + 1, it);
        }
    }

    if constexpr (SPLIT) {
        if (!fold_parts<T, TM, TN, NT>(acc, slices, done, smem_x)) return;
    }
    // four positions of one sample, 16-byte aligned
    const bool vec = sizeof(T) == 4 && g.ov % 4 == 0 && (reinterpret_cast<uintptr_t>(y) & 15) == 0;
#pragma unroll
    for (int h = 0; h < TN / 4; ++h) {
        const long long P = P0 + tile_col(tx, h);
        if (P >= g.P) return;
        uint32_t n, opos;
        g.d_ov.divmod((uint32_t)P, n, opos);
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            const int ol = o0 + ty * TM + i;
            if (ol >= g.Og) break;
            const int o = j * g.Og + ol;
            const T bv = bias != nullptr ? gload(bias + o) : (T)0;
            if (vec) {
                *reinterpret_cast<float4*>(y + ((size_t)n * g.O + o) * g.ov + opos) =
                    make_float4((float)(acc.at(i, 4 * h) + bv), (float)(acc.at(i, 4 * h + 1) + bv),
                                (float)(acc.at(i, 4 * h + 2) + bv), (float)(acc.at(i, 4 * h + 3) + bv));
                continue;
            }
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                if (P + t >= g.P) break;
                uint32_t nt, ot;
                g.d_ov.divmod((uint32_t)(P + t), nt, ot);
                y[((size_t)nt * g.O + o) * g.ov + ot] = acc.at(i, 4 * h + t) + bv;
            }
        }
    }
}

// grid.x: tiles of 16 * TN k'; grid.y: G * ceil(Og / BM); grid.z: slices of the position range.
template <typename T, int D, bool DEFORM, int V, int TM, int TN, int TY>
__global__ void __launch_bounds__(16 * TY, kCtasPerSm<T, TN, TY>)
exact_weight_kernel(const Geom g, const ExactGeom xg, const T* __restrict__ xcl, const Entry<T>* __restrict__ pts,
                    const T* __restrict__ dy, T* __restrict__ dwp, int chunks_per_slice) {
    constexpr int BM = TM * TY, BN = 16 * TN, NT = 16 * TY;
    constexpr int Q = BN / V, ALL = kBK * Q, ITEMS = (ALL + NT - 1) / NT, PAD = 16 / (int)sizeof(T);
    static_assert(NT % Q == 0 || Q % NT == 0, "a thread keeps its k' or alternates between whole blocks of them");
    extern __shared__ __align__(16) char smem_x[];
    T (*As)[kBK][BM + PAD] = reinterpret_cast<T (*)[kBK][BM + PAD]>(smem_x);
    T (*Bs)[kBK][BN] = reinterpret_cast<T (*)[kBK][BN]>(smem_x + 2 * kBK * (BM + PAD) * sizeof(T));
    const int tid = threadIdx.x, tx = tile_x(tid), ty = tile_y(tid);
    const int mt = (g.Og + BM - 1) / BM;
    const int j = blockIdx.y / mt, o0 = (blockIdx.y % mt) * BM;
    const T* xj = xcl + j * xg.Cg4;
    const long long chunks = (g.P + kBK - 1) / kBK;
    const long long ch0 = (long long)blockIdx.z * chunks_per_slice;
    const long long ch1 = ch0 + chunks_per_slice < chunks ? ch0 + chunks_per_slice : chunks;

    // Item it of a chunk: position row(it) of the chunk, k' krow(it).  Where a thread keeps its k' (KEEP) everything that
    // depends on it is computed once.
    constexpr bool KEEP = NT % Q == 0;
    constexpr int KN = KEEP ? 1 : ITEMS;
    auto row = [&](int it) { return (tid + it * NT) / Q; };
    uint32_t tap[KN], c[KN], k_ok = 0;
    const Entry<T>* pk[DEFORM ? KN : 1];
#pragma unroll
    for (int u = 0; u < KN; ++u) {
        const int kp = (int)blockIdx.x * BN + (tid + u * NT) % Q * V;
        if (kp < xg.Kp) k_ok |= 1u << u;
        xg.d_Cg4.divmod((uint32_t)(kp < xg.Kp ? kp : 0), tap[u], c[u]);
        if constexpr (DEFORM) pk[u] = pts + (size_t)(group_of(g, xg, j, c[u]) * g.kv + (int)tap[u]) * (size_t)g.P;
    }
    constexpr int kAhead = kAheadOf<T, D, DEFORM>, kStages = kAhead + 1;
    Sampler<T, D, DEFORM, V, NT> smp;
    smp.slots = smem_x + 2 * kBK * (BM + PAD + BN) * sizeof(T) + tid * V * sizeof(T);
    Entry<T> ent;
    T dv[TM];
    auto live = [&](long long ch, int it) {
        return (k_ok >> (KEEP ? 0 : it) & 1) && (ALL % NT == 0 || row(it) < kBK) && ch * kBK + row(it) < g.P;
    };
    auto fetch = [&](long long ch, int it) {
        if constexpr (DEFORM) {
            if (live(ch, it)) ent = load_entry(pk[KEEP ? 0 : it] + (ch * kBK + row(it)));
        }
    };
    auto issue = [&](int stage, long long ch, int it) {
        constexpr bool keep = KEEP;
        const bool ok = live(ch, it);
        const int u = keep ? 0 : it;
        int idx = -1;
        uint32_t n;
        const uint32_t P = ok ? (uint32_t)(ch * kBK + row(it)) : 0u;
        if constexpr (DEFORM) {
            n = g.d_ov.div(P);
        } else {
            const OutPos op = decompose_pos(g, P);
            n = (uint32_t)op.n;
            int at;
            if (locate_plain<D>(g, (int)tap[u], op, at)) idx = at;
        }
        smp.issue(g, xg, stage, xj + (size_t)n * ((uint32_t)g.iv * (uint32_t)xg.C4) + c[u], ent, ok, idx);
    };
    int fs = 0, is = 0;
    auto finish = [&](int buf, int it) {
        const Vec<T, V> r = smp.finish(fs);
        fs = fs + 1 == kStages ? 0 : fs + 1;
        if (ALL % NT != 0 && row(it) >= kBK) return;
        T* dst = &Bs[buf][row(it)][(tid + it * NT) % Q * V];
        if constexpr (V * sizeof(T) == 16) {
            uint4 w;
            memcpy(&w, &r, 16);
            *reinterpret_cast<uint4*>(dst) = w;
        } else {
#pragma unroll
            for (int v = 0; v < V; ++v) dst[v] = r.v[v];
        }
    };
    // dy: position tid % 16, output channels tid / 16 + TY * i
    auto load_dy = [&](long long ch) {
        const long long P = ch * kBK + tid % kBK;
        uint32_t n, opos;
        g.d_ov.divmod((uint32_t)(P < g.P ? P : 0), n, opos);
        const T* src = dy + ((size_t)n * g.O + (size_t)j * g.Og) * g.ov + opos;
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            const int o = o0 + tid / kBK + i * TY;
            dv[i] = (P < g.P && o < g.Og) ? gload(src + (size_t)o * g.ov) : (T)0;
        }
    };
    auto store_dy = [&](int buf) {
#pragma unroll
        for (int i = 0; i < TM; ++i) As[buf][tid % kBK][tid / kBK + i * TY] = dv[i];
    };

    Acc<T, TM, TN> acc;
    acc.clear();
    pdl_wait();
    if (ch0 < ch1) {
        long long ci = ch0, cf = ch0;                                 // chunks of the next item to issue / entry to fetch
        auto step = [&](int it) {
            smp.advance();
            if (ci < ch1) issue(is, ci, it);
            cp_async_commit();
            is = is + 1 == kStages ? 0 : is + 1;
            const int nf = (it + 1) % ITEMS;
            if (nf == 0) {
                ++ci;
                ++cf;
                if constexpr (DEFORM) {
                    // the entries a few chunks on come from DRAM: bring them to L2
                    const long long P = (cf + 3) * kBK + row(0);
                    if (KEEP && k_ok && cf + 3 < ch1 && P < g.P) asm volatile("prefetch.global.L2 [%0];" ::"l"(pk[0] + P));
                }
            }
            if (cf < ch1) fetch(cf, nf);
        };
        load_dy(ch0);
        fetch(ch0, 0);
#pragma unroll
        for (int i = 0; i < kAhead; ++i) step(i % ITEMS);
#pragma unroll
        for (int it = 0; it < ITEMS; ++it) {
            step((it + kAhead) % ITEMS);
            cp_async_wait_group<kAhead>();
            finish(0, it);
        }
        store_dy(0);
        for (long long ch = ch0; ch < ch1; ++ch) {
            const int buf = (int)(ch - ch0) & 1;
            __syncthreads();
            const bool more = ch + 1 < ch1;
            if (more) load_dy(ch + 1);
#pragma unroll
            for (int it = 0; it < ITEMS; ++it) {
                step((it + kAhead) % ITEMS);
#pragma unroll
                for (int kk = it * kBK / ITEMS; kk < (it + 1) * kBK / ITEMS; ++kk)
                    tile_step<T, TM, TN>(acc, As[buf][kk], Bs[buf][kk], tx, ty, 0);
                cp_async_wait_group<kAhead>();
                if (more) finish(buf ^ 1, it);
            }
            if (more) store_dy(buf ^ 1);
        }
    }
    pdl_trigger();
#pragma unroll
    for (int h = 0; h < TN / 4; ++h) {
        const int k0 = blockIdx.x * BN + tile_col(tx, h);
        if (k0 >= xg.Kp64) return;
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            const int ol = o0 + ty * TM + i;
            if (ol >= g.Og) break;
            T* dst = dwp + ((size_t)blockIdx.z * g.O + j * g.Og + ol) * xg.Kp64 + k0;
#pragma unroll
            for (int t = 0; t < 4; ++t) dst[t] = acc.at(i, 4 * h + t);
        }
    }
}

// ------------------------------------------------------------------------------------------------------------------
// Backward data.  grid.x: tiles of BN positions; grid.y: G * Kp64 / 64.  A thread holds four consecutive k' rows (whole
// vectors of channels of one tap) at TN consecutive positions; the lanes of a warp cover 32 k' at four position runs, so
// the corner vectors of a position are one contiguous run of the channels-last tensors.  Per (vector, position): corner
// dot products sum_c col_c * x_c -- combined by the interpolation gradient, which is linear in them -- and one
// reduction per corner into dxcl.  The offset terms of the tile are summed over its channel vectors in shared memory;
// where a tile holds whole segments (PLAIN) the sums are the offset gradient and are stored, else added to a zeroed one.
// ------------------------------------------------------------------------------------------------------------------
// interp_grad() of corner dot products, factored: differences along the axis first, then the weights of the others.
template <typename T, int D>
__device__ __forceinline__ void dot_grad(const Pt<T, D>& s, const T (&d)[1 << D], T (&gr)[D]) {
    if constexpr (D == 2) {
        gr[0] = (d[2] - d[0]) * s.hw[1] + (d[3] - d[1]) * s.lw[1];
        gr[1] = (d[1] - d[0]) * s.hw[0] + (d[3] - d[2]) * s.lw[0];
    } else {
        const T *hw = s.hw, *lw = s.lw;
        gr[0] = ((d[4] - d[0]) * hw[2] + (d[5] - d[1]) * lw[2]) * hw[1] + ((d[6] - d[2]) * hw[2] + (d[7] - d[3]) * lw[2]) * lw[1];
        gr[1] = ((d[2] - d[0]) * hw[2] + (d[3] - d[1]) * lw[2]) * hw[0] + ((d[6] - d[4]) * hw[2] + (d[7] - d[5]) * lw[2]) * lw[0];
        gr[2] = ((d[1] - d[0]) * hw[1] + (d[3] - d[2]) * lw[1]) * hw[0] + ((d[5] - d[4]) * hw[1] + (d[7] - d[6]) * lw[1]) * lw[0];
    }
}

template <typename T, int V>
constexpr int kDataTn = sizeof(T) == 4 && V == 4 ? 8 : (sizeof(T) == 8 && V == 1 ? 1 : 2);

template <typename T, int D, bool DEFORM, int V>
__global__ void __launch_bounds__(kXThreads, sizeof(T) == 4 ? 2 : 1)
exact_data_kernel(const Geom g, const ExactGeom xg, const T* __restrict__ xcl, const Entry<T>* __restrict__ pts,
                  const T* __restrict__ wt, const T* __restrict__ dy, T* __restrict__ dxcl, T* __restrict__ doff,
                  const int plain) {
    constexpr int BM = 64, TM = 4, TN = kDataTn<T, V>, BN = 16 * TN, L16 = 16 / (int)sizeof(T);
    constexpr int NV = TM / V, NG = BM / V, DY = kBK * BN / kXThreads;
    constexpr int kMain = 2 * kBK * (BM + BN), kEpi = DEFORM ? D * NG * BN : 0;
    __shared__ __align__(16) T smem[kMain > kEpi ? kMain : kEpi];
    __shared__ int key_s[NG];
    T (*As)[kBK][BM] = reinterpret_cast<T (*)[kBK][BM]>(smem);
    T (*Bs)[kBK][BN] = reinterpret_cast<T (*)[kBK][BN]>(smem + 2 * kBK * BM);
    const int tid = threadIdx.x, tx = tile_x(tid), ty = tile_y(tid);
    const int mt = xg.Kp64 / BM;
    const int j = blockIdx.y / mt, m0 = (blockIdx.y % mt) * BM;
    const long long P0 = (long long)blockIdx.x * BN;

    // the dy column this thread brings in: position tid % BN, output channels tid / BN + i * (256 / BN)
    const long long Pb = P0 + tid % BN;
    uint32_t nb = 0, oposb = 0;
    if (Pb < g.P) g.d_ov.divmod((uint32_t)Pb, nb, oposb);
    const T* dyb = dy + ((size_t)nb * g.O + (size_t)j * g.Og) * g.ov + oposb;
    const T* wg = wt + (size_t)j * g.Og * xg.Kp64 + m0;
    T dv[DY];
    auto load = [&](int ch) {
#pragma unroll
        for (int i = 0; i < kBK * BM / L16 / kXThreads; ++i) {
            const int e = tid + i * kXThreads, row = e / (BM / L16), m = (e % (BM / L16)) * L16;
            const bool ok = ch * kBK + row < g.Og;
            cp_async16(&As[ch & 1][row][m], wg + (size_t)(ok ? ch * kBK + row : 0) * xg.Kp64 + m, ok);
        }
#pragma unroll
        for (int i = 0; i < DY; ++i) {
            const int o = ch * kBK + tid / BN + i * (kXThreads / BN);
            dv[i] = (Pb < g.P && o < g.Og) ? gload(dyb + (size_t)o * g.ov) : (T)0;
        }
    };
    auto store = [&](int ch) {
#pragma unroll
        for (int i = 0; i < DY; ++i) Bs[ch & 1][tid / BN + i * (kXThreads / BN)][tid % BN] = dv[i];
    };

    Acc<T, TM, TN> acc;
    acc.clear();
    const int nch = (g.Og + kBK - 1) / kBK;
    pdl_wait();
    load(0);
    store(0);
    for (int ch = 0; ch < nch; ++ch) {
        cp_async_wait();
        __syncthreads();
        if (ch + 1 < nch) load(ch + 1);
#pragma unroll
        for (int kk = 0; kk < kBK; ++kk) {
            T a[TM], b[TN];
            load_row<T, TM>(&As[ch & 1][kk][tx * TM], a);
            load_row<T, TN>(&Bs[ch & 1][kk][ty * TN], b);
            acc.fma(a, b);
        }
        if (ch + 1 < nch) store(ch + 1);
    }

    // ---- epilogue: acc.at(r, i) = col[m0 + tx*4 + r, P0 + ty*TN + i] ----
    uint32_t tap[NV], c[NV];
    int key[NV];
#pragma unroll
    for (int u = 0; u < NV; ++u) {
        const int kp = m0 + tx * TM + u * V;
        key[u] = -1;
        tap[u] = c[u] = 0;
        if (kp < xg.Kp) {
            xg.d_Cg4.divmod((uint32_t)kp, tap[u], c[u]);
            key[u] = (DEFORM ? group_of(g, xg, j, c[u]) : 0) * g.kv + (int)tap[u];
        }
    }
    T (*con)[NG][BN] = reinterpret_cast<T (*)[NG][BN]>(smem);
    pdl_trigger();
    if constexpr (DEFORM) {
        __syncthreads();                                   // the operand tiles are done with
        if (ty == 0) {                                     // (two warps hold such threads: all sixteen tx)
#pragma unroll
            for (int u = 0; u < NV; ++u) key_s[tx * NV + u] = key[u];
        }
    }
#pragma unroll
    for (int i = 0; i < TN; ++i) {
        const long long P = P0 + ty * TN + i;
        const bool pok = P < g.P;
        OutPos op;
        if constexpr (DEFORM) op.n = (int)g.d_ov.div((uint32_t)(pok ? P : 0));
        else op = decompose_pos(g, pok ? P : 0);
        const size_t nbase = (size_t)op.n * g.iv * xg.C4 + j * xg.Cg4;
#pragma unroll
        for (int u = 0; u < NV; ++u) {
            using Ln = Lanes<T, V>;
            T col[V];
#pragma unroll
            for (int v = 0; v < V; ++v) col[v] = acc.at(u * V + v, i);
            typename Ln::L lcol[Ln::N];
            Ln::load(col, lcol);
            if constexpr (DEFORM) {
                T gr[D];
#pragma unroll
                for (int a = 0; a < D; ++a) gr[a] = (T)0;
                if (pok && key[u] >= 0) {
                    const Entry<T> e = load_entry(pts + (size_t)key[u] * (size_t)g.P + (size_t)P);
                    if (!(e.bits >> 31)) {
                        Pt<T, D> s;
                        entry_weights<T, D>(e, s);
                        uint32_t at[1 << D];
                        entry_corners<D>(g, xg, e.bits, at);
                        if (doff != nullptr) {
                            const T* xn = xcl + nbase + c[u];
                            Vec<T, V> cv[1 << D];
#pragma unroll
                            for (int k = 0; k < (1 << D); ++k) cv[k] = load_vec<T, V>(xn + at[k]);
                            T dot[1 << D];
#pragma unroll
                            for (int k = 0; k < (1 << D); ++k) {
                                typename Ln::L x[Ln::N];
                                Ln::load(cv[k].v, x);
#pragma unroll
                                for (int v = 0; v < Ln::N; ++v) x[v] = Ln::mul(lcol[v], x[v]);
                                dot[k] = Ln::sum(x);
                            }
                            dot_grad<T, D>(s, dot, gr);
                        }
                        if (dxcl != nullptr) {
                            T cw[1 << D];
                            corner_weights<T, D>(s, cw);
                            T* dn = dxcl + nbase + c[u];
#pragma unroll
                            for (int k = 0; k < (1 << D); ++k) {
                                typename Ln::L p[Ln::N];
                                const auto wk = Ln::same(cw[k]);
#pragma unroll
                                for (int v = 0; v < Ln::N; ++v) p[v] = Ln::mul(wk, lcol[v]);
                                T wv[V];
                                Ln::store(p, wv);
                                add_vec<T, V>(dn + at[k], wv);
                            }
                        }
                    } else if (D == 3 && g.oob) {
                        T mag = (T)0;
#pragma unroll
                        for (int v = 0; v < V; ++v) mag += col[v] > (T)0 ? col[v] : -col[v];
#pragma unroll
                        for (int a = 0; a < D; ++a)
                            gr[a] = (e.bits & (1u << (2 * a))) ? -mag : ((e.bits & (2u << (2 * a))) ? mag : (T)0);
                    }
                }
                if (doff != nullptr) {
#pragma unroll
                    for (int a = 0; a < D; ++a) con[a][tx * NV + u][ty * TN + i] = gr[a];
                }
            } else {
                int idx;
                if (dxcl != nullptr && pok && key[u] >= 0 && locate_plain<D>(g, (int)tap[u], op, idx))
                    add_vec<T, V>(dxcl + nbase + c[u] + (size_t)idx * xg.C4, col);
            }
        }
    }
    if constexpr (DEFORM) {
        if (doff == nullptr) return;
        __syncthreads();
        if (Pb >= g.P) return;
        T* dn = doff + (size_t)nb * g.dg * g.kv * D * g.ov + oposb;
        for (int a = tid / BN; a < D; a += kXThreads / BN) {
            int run = -1;
            T sum = (T)0;
            for (int r = 0; r <= NG; ++r) {
                const int kr = r < NG ? key_s[r] : -2;
                if (kr != run) {
                    if (run >= 0) {
                        T* dst = dn + ((size_t)run * D + a) * g.ov;
                        if (plain) *dst = sum;
                        else atomicAdd(dst, sum);
                    }
                    run = kr;
                    sum = (T)0;
                }
                if (r < NG) sum += con[a][r][tid % BN];
            }
        }
    }
}

// ------------------------------------------------------------------------------------------------------------------
// Epilogue of a backward pass, one launch: dxcl -> dX (tiled transpose) and the weight slices -> dW.
// ------------------------------------------------------------------------------------------------------------------
template <typename T>
struct FoldArgs {
    const T *dxcl, *dwp;
    T *dx, *dw;
    unsigned nx, tx, ty;             // blocks of the transpose, its tiles along positions / channels
    int slices, add;                 // add: accumulate into dX and dW
};

template <typename T>
__global__ void __launch_bounds__(kXThreads)
exact_fold_kernel(const Geom g, const ExactGeom xg, const FoldArgs<T> a) {
    constexpr int TC = kCopyTile<T>;
    __shared__ T tile[TC][TC + 1];
    pdl_wait();
    unsigned b = blockIdx.x;
    if (b < a.nx) {
        const unsigned px = b % a.tx, r = b / a.tx, cy = r % a.ty, n = r / a.ty;
        const int tx = threadIdx.x % 32, ty = threadIdx.x / 32;
        const int p0 = (int)px * TC, c0 = (int)cy * TC;
        const T* in = a.dxcl + (size_t)n * g.iv * xg.C4;
        T v[TC / 8][TC / 32];
#pragma unroll
        for (int i = 0; i < TC / 8; ++i) {
            const int p = p0 + ty + i * 8;
#pragma unroll
            for (int h = 0; h < TC / 32; ++h) {
                const int c4 = c0 + h * 32 + tx;
                v[i][h] = (p < g.iv && c4 < xg.C4) ? gload(in + (size_t)p * xg.C4 + c4) : (T)0;
            }
        }
#pragma unroll
        for (int i = 0; i < TC / 8; ++i)
#pragma unroll
            for (int h = 0; h < TC / 32; ++h) tile[ty + i * 8][h * 32 + tx] = v[i][h];
        __syncthreads();
#pragma unroll
        for (int i = 0; i < TC / 8; ++i) {
            const int c4 = c0 + ty + i * 8;
            uint32_t seg, r4;
            xg.d_S4.divmod((uint32_t)c4, seg, r4);
            if (c4 >= xg.C4 || (int)r4 >= xg.S) continue;
            T* dst = a.dx + ((size_t)n * g.C + seg * xg.S + r4) * g.iv;
#pragma unroll
            for (int h = 0; h < TC / 32; ++h) {
                const int p = p0 + h * 32 + tx;
                if (p < g.iv) dst[p] = a.add ? dst[p] + tile[h * 32 + tx][ty + i * 8] : tile[h * 32 + tx][ty + i * 8];
            }
        }
        return;
    }
    b -= a.nx;
    const uint32_t e = b * kXThreads + threadIdx.x;                    // [O][Kp], k' fastest: coalesced slices
    uint32_t o, kp;
    xg.d_Kp64.divmod(e, o, kp);
    if ((int)o >= g.O || (int)kp >= xg.Kp) return;
    uint32_t tap, c4, seg, r4;
    xg.d_Cg4.divmod(kp, tap, c4);
    xg.d_S4.divmod(c4, seg, r4);
    if ((int)r4 >= xg.S) return;
    const size_t step = (size_t)g.O * xg.Kp64;
    const T* src = a.dwp + (size_t)o * xg.Kp64 + kp;
    T s = (T)0;
#pragma unroll 4
    for (int i = 0; i < a.slices; ++i) s += gload(src + i * step);
    T* dst = a.dw + ((size_t)o * g.Cg + seg * xg.S + r4) * g.kv + tap;
    *dst = a.add ? *dst + s : s;
}

// ------------------------------------------------------------------------------------------------------------------
// Host side
// ------------------------------------------------------------------------------------------------------------------
size_t up256(size_t v) { return (v + 255) / 256 * 256; }

// channels of a vector: 16 bytes' worth, except where a segment is so short that most of the vector would be padding
int vec_width(const Geom& g, int dtype, int S) {
    (void)g;
    if (dtype == 1) return S >= 2 ? 2 : 1;
    return S >= 3 ? 4 : 1;
}

ExactGeom exact_geom(const Geom& g, int dtype) {
    ExactGeom x;
    x.S = g.cpg < g.Cg ? g.cpg : g.Cg;
    x.split = g.cpg > g.Cg ? 1 : 0;
    x.segs = g.Cg / x.S;
    const int v = vec_width(g, dtype, x.S);
    x.S4 = (x.S + v - 1) / v * v;
    x.Cg4 = x.segs * x.S4;
    x.C4 = g.G * x.Cg4;
    x.Kp = g.kv * x.Cg4;
    x.Kp16 = (x.Kp + 15) / 16 * 16;
    x.Kp64 = (x.Kp + 63) / 64 * 64;
    x.Og4 = (g.Og + 3) / 4 * 4;
    x.d_Cg4.init(x.Cg4); x.d_S4.init(x.S4); x.d_Og4.init(x.Og4); x.d_Kp64.init(x.Kp64);
    return x;
}

// Tiles of the forward and weight kernels: heights of 32, 64, 96 or 128 output channels where they are wide (64 or 128
// with single-channel vectors), 32 or 64 where narrow; the whole group where it has at most the largest, else equal
// parts.  Wide from 600 warp pairs' worth of tiles up (128 positions x 8 channels each; B200, GPU time of forward and
// backward weight: 6272 positions x 128 channels, 784: 56 us wide, 85 us narrow; 8192 x 32, 256: narrow a third faster).
struct ExactTiles {
    int wide, tm, tn, ty, mt, bn;
    long long slots;                 // CTAs that run at once
};
ExactTiles exact_tiles(const Geom& g, const ExactGeom& x, int dtype) {
    ExactTiles t;
    t.wide = dtype == 0 && (g.P + 127) / 128 * g.G * ((g.Og + 31) / 32 * 4) >= 600;
    const int most = t.wide ? 128 : 64;
    t.mt = (g.Og + most - 1) / most;
    int rows = ((g.Og + t.mt - 1) / t.mt + 31) / 32 * 32;
    if (t.wide && vec_width(g, dtype, x.S) == 1) rows = (rows + 63) / 64 * 64;
    t.tn = t.wide ? 8 : 4;
    t.ty = t.wide ? rows / 8 : 16;
    t.tm = rows / t.ty;
    t.bn = 16 * t.tn;
    const int per_sm = dtype == 1 ? 1 : (!t.wide ? 2 : (t.ty == 4 ? 5 : (t.ty == 8 ? 3 : (t.ty == 12 ? 2 : 1))));
    t.slots = (long long)sm_count() * per_sm;
    return t;
}

// The number of parts (up to `most`) whose CTAs fill whole waves best; of equally good ones the first, because every
// part writes partial sums.
long long best_parts(long long tiles, long long slots, long long most) {
    long long s = 1;
    double best = 0.0;
    for (long long k = 1; k <= most; ++k) {
        const double waves = (double)(tiles * k) / (double)slots;
        const double fill = waves / (double)(long long)(waves + 0.999999);
        if (fill > best + 0.02) { best = fill; s = k; }
    }
    return s;
}

// Slices of the position range in the weight pass: up to three waves, none under 4 chunks.
int weight_slices(const Geom& g, const ExactGeom& x, int dtype, int& per) {
    const long long chunks = (g.P + kBK - 1) / kBK;
    const ExactTiles t = exact_tiles(g, x, dtype);
    const long long tiles = (long long)((x.Kp + t.bn - 1) / t.bn) * g.G * t.mt;
    long long most = 3 * t.slots / tiles;
    if (most > chunks / 4) most = chunks / 4;
    if (most > 256) most = 256;
    const long long s = best_parts(tiles, t.slots, most);
    per = (int)((chunks + s - 1) / s);
    return (int)((chunks + per - 1) / per);
}

// Parts of the K range in the forward pass: only within the first wave, none under 3 chunks.
int forward_parts(const Geom& g, const ExactGeom& x, int dtype, int& per) {
    const int chunks = x.Kp16 / kBK;
    const ExactTiles t = exact_tiles(g, x, dtype);
    const long long tiles = (g.P + t.bn - 1) / t.bn * g.G * t.mt;
    long long most = t.slots / tiles;
    if (most > chunks / 3) most = chunks / 3;
    const long long s = best_parts(tiles, t.slots, most);
    per = (int)((chunks + s - 1) / s);
    return (chunks + per - 1) / per;
}

struct ExactLayout {
    size_t xcl, wk, pts, dxcl, dwp, slices, done, done_n, total;     // done_n: counters
};
ExactLayout exact_layout(const Geom& g, const ExactGeom& x, int dtype, int deform, int pass) {
    const size_t es = dtype == 1 ? 8 : 4;
    ExactLayout l;
    size_t at = 0;
    l.xcl = at; at += up256((size_t)g.N * g.iv * x.C4 * es);
    l.wk = at; at += up256((size_t)g.G * (pass == 0 ? (size_t)x.Kp16 * x.Og4 : (size_t)g.Og * x.Kp64) * es);
    l.pts = at; at += deform ? up256((size_t)g.dg * g.kv * g.P * (dtype == 1 ? sizeof(Entry<double>) : sizeof(Entry<float>))) : 0;
    l.dxcl = at; l.dwp = at; l.slices = at; l.done = at; l.done_n = 0;
    if (pass == 0) {
        int per;
        const int parts = forward_parts(g, x, dtype, per);
        if (parts > 1) {             // no more CTAs than run at once: at most 14 MB
            const ExactTiles t = exact_tiles(g, x, dtype);
            l.done_n = (size_t)((g.P + t.bn - 1) / t.bn) * g.G * t.mt;
            at += up256(l.done_n * parts * (size_t)(t.tm * t.ty) * t.bn * es);
            l.done = at;
            at += up256(l.done_n * sizeof(unsigned));
        }
    }
    if (pass == 1 || pass == 3) { l.dxcl = at; at += up256((size_t)g.N * g.iv * x.C4 * es); }
    if (pass == 2 || pass == 3) {
        int per;
        l.dwp = at;
        at += up256((size_t)weight_slices(g, x, dtype, per) * g.O * x.Kp64 * es);
    }
    l.total = at;
    return l;
}

template <typename T, int D>
int launch_prep(const Geom& g, const ExactGeom& x, PrepArgs<T> a, cudaStream_t st) {
    a.nb = a.dbias != nullptr ? (unsigned)g.O : 0u;
    a.nx = a.np = a.nw = a.nz = 0;
    a.bpk = 1;
    a.tx = (unsigned)((g.iv + kCopyTile<T> - 1) / kCopyTile<T>);
    a.ty = (unsigned)((x.C4 + kCopyTile<T> - 1) / kCopyTile<T>);
    if (a.xcl != nullptr) a.nx = a.tx * a.ty * (unsigned)g.N;
    if (a.pts != nullptr) {
        a.bpk = (unsigned)((g.P + kPtsPerThread * kXThreads - 1) / (kPtsPerThread * kXThreads));
        a.np = a.bpk * (unsigned)(g.dg * g.kv);
    }
    if (a.wk != nullptr) {
        const size_t n = (size_t)g.G * (a.backward ? (size_t)g.Og * x.Kp64 : (size_t)x.Kp16 * x.Og4);
        a.nw = (unsigned)((n + 4 * kXThreads - 1) / (4 * kXThreads));
    }
    if (a.zero != nullptr) a.nz = (unsigned)((a.zero_n * sizeof(T) + 64 * kXThreads - 1) / (64 * kXThreads));
    const unsigned nz2 = a.zero2 != nullptr ? (unsigned)((a.zero2_n * sizeof(T) + 64 * kXThreads - 1) / (64 * kXThreads)) : 0u;
    const unsigned blocks = a.nb + a.nx + a.np + a.nw + a.nz + nz2;
    if (blocks == 0) return 0;
    return launch_dependent(exact_prep_kernel<T, D>, dim3(blocks), dim3(kXThreads), 0, st, g, x, a) == cudaSuccess ? 0 : -5;
}

template <typename K>
bool allow_smem(K kernel, int bytes) {
    return bytes <= 48 * 1024 || cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess;
}

template <typename T, int D, bool DEFORM, int V, int TM, int TN, int TY>
int launch_forward(const Geom& g, const ExactGeom& x, dim3 grid, const T* xcl, const Entry<T>* pts, const T* w2,
                   const T* bias, T* y, int per, T* slices, unsigned* done, cudaStream_t st) {
    auto kernel = grid.z > 1 ? exact_forward_kernel<T, D, DEFORM, V, TM, TN, TY, true>
                             : exact_forward_kernel<T, D, DEFORM, V, TM, TN, TY, false>;
    const int smem = 2 * kBK * (TM * TY + 16 * TN) * (int)sizeof(T) + Sampler<T, D, DEFORM, V, 16 * TY>::kBytes;
    if (!allow_smem(kernel, smem)) return -5;
    return launch_dependent(kernel, grid, dim3(16 * TY), smem, st, g, x, xcl, pts, w2, bias, y, per, slices, done) == cudaSuccess
               ? 0 : -5;
}

template <typename T, int D, bool DEFORM, int V, int TM, int TN, int TY>
int launch_weight(const Geom& g, const ExactGeom& x, dim3 grid, const T* xcl, const Entry<T>* pts, const T* dy, T* dwp,
                  int per, cudaStream_t st) {
    auto kernel = exact_weight_kernel<T, D, DEFORM, V, TM, TN, TY>;
    const int smem = 2 * kBK * (TM * TY + 16 / (int)sizeof(T) + 16 * TN) * (int)sizeof(T) + Sampler<T, D, DEFORM, V, 16 * TY>::kBytes;
    if (!allow_smem(kernel, smem)) return -5;
    return launch_dependent(kernel, grid, dim3(16 * TY), smem, st, g, x, xcl, pts, dy, dwp, per) == cudaSuccess ? 0 : -5;
}

// FN<T, D, DEFORM, V, TM, TN, TY> with the tile that exact_tiles() chose
#define DCN_EXACT_TILE(FN, ...)                                                                        \
    do {                                                                                               \
        if constexpr (std::is_same<T, float>::value) {                                                 \
            if (t.wide && t.ty == 8) return FN<T, D, DEFORM, V, 8, 8, 8>(__VA_ARGS__);                 \
            if (t.wide && t.ty == 16) return FN<T, D, DEFORM, V, 8, 8, 16>(__VA_ARGS__);               \
            if constexpr (V > 1) {                                                                     \
                if (t.wide && t.ty == 4) return FN<T, D, DEFORM, V, 8, 8, 4>(__VA_ARGS__);             \
                if (t.wide && t.ty == 12) return FN<T, D, DEFORM, V, 8, 8, 12>(__VA_ARGS__);           \
            }                                                                                          \
        }                                                                                              \
        if (t.tm == 2) return FN<T, D, DEFORM, V, 2, 4, 16>(__VA_ARGS__);                              \
        return FN<T, D, DEFORM, V, 4, 4, 16>(__VA_ARGS__);                                             \
    } while (0)

template <typename T, int D, bool DEFORM, int V>
int pick_forward(const ExactTiles& t, const Geom& g, const ExactGeom& x, dim3 grid, const T* xcl, const Entry<T>* pts,
                 const T* w2, const T* bias, T* y, int per, T* slices, unsigned* done, cudaStream_t st) {
    DCN_EXACT_TILE(launch_forward, g, x, grid, xcl, pts, w2, bias, y, per, slices, done, st);
}
template <typename T, int D, bool DEFORM, int V>
int pick_weight(const ExactTiles& t, const Geom& g, const ExactGeom& x, dim3 grid, const T* xcl, const Entry<T>* pts,
                const T* dy, T* dwp, int per, cudaStream_t st) {
    DCN_EXACT_TILE(launch_weight, g, x, grid, xcl, pts, dy, dwp, per, st);
}

template <typename T, int D, bool DEFORM, int V>
int run_forward(const Geom& g, const ExactGeom& x, const void* x_in, const void* off, const void* w, const void* bias,
                void* y, uint8_t* ws, cudaStream_t st) {
    const int dtype = sizeof(T) == 8;
    const ExactLayout l = exact_layout(g, x, dtype, DEFORM, 0);
    PrepArgs<T> a = {};
    a.x = (const T*)x_in; a.off = (const T*)off; a.w = (const T*)w;
    a.xcl = (T*)(ws + l.xcl); a.wk = (T*)(ws + l.wk);
    a.pts = DEFORM ? (Entry<T>*)(ws + l.pts) : nullptr;
    int per;
    const int parts = forward_parts(g, x, dtype, per);
    if (parts > 1) {
        a.zero = (T*)(ws + l.done);
        a.zero_n = (l.done_n * sizeof(unsigned) + sizeof(T) - 1) / sizeof(T);
    }
    const int r = launch_prep<T, D>(g, x, a, st);
    if (r != 0) return r;
    const ExactTiles t = exact_tiles(g, x, dtype);
    const dim3 grid((unsigned)((g.P + t.bn - 1) / t.bn), (unsigned)(g.G * t.mt), (unsigned)parts);
    return pick_forward<T, D, DEFORM, V>(t, g, x, grid, a.xcl, a.pts, a.wk, (const T*)bias, (T*)y, per, (T*)(ws + l.slices),
                                         (unsigned*)(ws + l.done), st);
}

// pass 1: backward data, 2: backward weight, 3: both.  add: dX and dW accumulate (else they are overwritten).
template <typename T, int D, bool DEFORM, int V>
int run_backward(const Geom& g, const ExactGeom& x, int pass, int add, const void* x_in, const void* off, const void* w,
                 const void* dy, void* dx, void* doff, void* dw, void* db, uint8_t* ws, cudaStream_t st) {
    const int dtype = sizeof(T) == 8;
    const ExactLayout l = exact_layout(g, x, dtype, DEFORM, pass);
    const bool data = dx != nullptr || (DEFORM && doff != nullptr);
    PrepArgs<T> a = {};
    a.backward = 1;
    a.x = (const T*)x_in; a.off = (const T*)off; a.w = (const T*)w; a.dy = (const T*)dy;
    a.dbias = (T*)db;
    a.xcl = (DEFORM || dw != nullptr) ? (T*)(ws + l.xcl) : nullptr;
    a.pts = DEFORM ? (Entry<T>*)(ws + l.pts) : nullptr;
    a.wk = data ? (T*)(ws + l.wk) : nullptr;
    a.zero = dx != nullptr ? (T*)(ws + l.dxcl) : nullptr;
    a.zero_n = (size_t)g.N * g.iv * x.C4;
    // a 64-row tile of the data kernel holds whole segments: its offset sums are the offset gradient, else parts of it
    const int plain = x.S4 <= 64 && 64 % x.S4 == 0 && !x.split;
    if (DEFORM && doff != nullptr && !plain) {
        a.zero2 = (T*)doff;
        a.zero2_n = (size_t)g.N * g.dg * g.kv * D * g.ov;
    }
    int r = launch_prep<T, D>(g, x, a, st);
    if (r != 0) return r;
    if (data) {
        constexpr int BN = 16 * kDataTn<T, V>;
        const dim3 grid((unsigned)((g.P + BN - 1) / BN), (unsigned)(g.G * (x.Kp64 / 64)));
        if (launch_dependent(exact_data_kernel<T, D, DEFORM, V>, grid, dim3(kXThreads), 0, st, g, x, a.xcl, a.pts, a.wk,
                             (const T*)dy, a.zero, DEFORM ? (T*)doff : nullptr, plain) != cudaSuccess)
            return -5;
    }
    FoldArgs<T> f = {};
    f.add = add;
    if (dw != nullptr) {
        int per;
        f.slices = weight_slices(g, x, dtype, per);
        f.dwp = (T*)(ws + l.dwp);
        f.dw = (T*)dw;
        const ExactTiles t = exact_tiles(g, x, dtype);
        const dim3 grid((unsigned)((x.Kp + t.bn - 1) / t.bn), (unsigned)(g.G * t.mt), (unsigned)f.slices);
        r = pick_weight<T, D, DEFORM, V>(t, g, x, grid, a.xcl, a.pts, (const T*)dy, (T*)(ws + l.dwp), per, st);
        if (r != 0) return r;
    }
    f.tx = (unsigned)((g.iv + kCopyTile<T> - 1) / kCopyTile<T>);
    f.ty = (unsigned)((x.C4 + kCopyTile<T> - 1) / kCopyTile<T>);
    if (dx != nullptr) {
        f.dxcl = a.zero;
        f.dx = (T*)dx;
        f.nx = f.tx * f.ty * (unsigned)g.N;
    }
    const unsigned blocks = f.nx + (dw != nullptr ? (unsigned)(((size_t)g.O * x.Kp64 + kXThreads - 1) / kXThreads) : 0u);
    if (blocks > 0) {
        if (launch_dependent(exact_fold_kernel<T>, dim3(blocks), dim3(kXThreads), 0, st, g, x, f) != cudaSuccess) return -5;
    }
    return 0;
}

#define DCN_EXACT_V(FN, T, D, DEF, ...)                                                          \
    do {                                                                                         \
        const int v = vec_width(g, sizeof(T) == 8, x.S);                                         \
        if constexpr (sizeof(T) == 8) {                                                          \
            if (v == 2) return FN<T, D, DEF, 2>(__VA_ARGS__);                                    \
            return FN<T, D, DEF, 1>(__VA_ARGS__);                                                \
        } else {                                                                                 \
            if (v == 4) return FN<T, D, DEF, 4>(__VA_ARGS__);                                    \
            return FN<T, D, DEF, 1>(__VA_ARGS__);                                                \
        }                                                                                        \
    } while (0)
#define DCN_EXACT_D(FN, T, ...)                                                                  \
    do {                                                                                         \
        if (ndim == 2) {                                                                         \
            if (deform) DCN_EXACT_V(FN, T, 2, true, __VA_ARGS__);                                \
            else DCN_EXACT_V(FN, T, 2, false, __VA_ARGS__);                                      \
        } else {                                                                                 \
            if (deform) DCN_EXACT_V(FN, T, 3, true, __VA_ARGS__);                                \
            else DCN_EXACT_V(FN, T, 3, false, __VA_ARGS__);                                      \
        }                                                                                        \
    } while (0)

}  // namespace

// Problems these kernels take: uniform segments, index ranges of the point entries and 32-bit element offsets.
bool exact_supported(const Geom& g, int dtype, int deform) {
    if (g.cl) return false;
    if (deform && g.Cg % g.cpg != 0 && g.cpg % g.Cg != 0) return false;
    const ExactGeom x = exact_geom(g, dtype);
    if (g.iv >= (1 << 28)) return false;
    if ((long long)x.C4 * g.iv >= (1ll << 31) || (long long)g.O * x.Kp64 >= (1ll << 31)) return false;
    if ((long long)x.Kp16 * x.Og4 * g.G >= (1ll << 31)) return false;
    const long long rows = (long long)g.G * ((g.Og + 31) / 32), cols = (long long)g.G * (x.Kp64 / 64);
    if (rows > 65535 || cols > 65535) return false;
    const long long blocks = ((long long)g.iv / 32 + 1) * (x.C4 / 32 + 1) * g.N + (g.P / kXThreads + 1) * (long long)g.dg * g.kv;
    return blocks < (1ll << 30);
}

size_t exact_workspace_bytes(const Geom& g, int dtype, int deform, int pass) {
    return exact_layout(g, exact_geom(g, dtype), dtype, deform, pass).total;
}

int exact_launch_count(int pass) { return pass == 0 ? 2 : (pass == 3 ? 4 : 3); }

int exact_forward(const Geom& g, int dtype, int ndim, int deform, const void* x_in, const void* off, const void* w,
                  const void* bias, void* y, void* ws, cudaStream_t st) {
    const ExactGeom x = exact_geom(g, dtype);
    uint8_t* b = (uint8_t*)ws;
    if (dtype == 0) DCN_EXACT_D(run_forward, float, g, x, x_in, off, w, bias, y, b, st);
    DCN_EXACT_D(run_forward, double, g, x, x_in, off, w, bias, y, b, st);
}

int exact_backward(const Geom& g, int dtype, int ndim, int deform, int pass, int add, const void* x_in, const void* off,
                   const void* w, const void* dy, void* dx, void* doff, void* dw, void* db, void* ws, cudaStream_t st) {
    const ExactGeom x = exact_geom(g, dtype);
    uint8_t* b = (uint8_t*)ws;
    if (dtype == 0) DCN_EXACT_D(run_backward, float, g, x, pass, add, x_in, off, w, dy, dx, doff, dw, db, b, st);
    DCN_EXACT_D(run_backward, double, g, x, pass, add, x_in, off, w, dy, dx, doff, dw, db, b, st);
}

}  // namespace dcn
