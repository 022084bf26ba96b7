// BF16 tensor-core path of libdcn (sm_100a): implicit-GEMM kernels on tcgen05 with accumulators in tensor
// memory.  fp32 tensors in and out; sampled patches, weights and output gradients are rounded to bf16 on
// their way into shared memory; coordinates, interpolation weights and accumulation stay fp32.
//
// Replaces, without ever materialising the reference's column buffer:
//   forward          deformable_im2col + SGEMM       (deform3d/lib/deform_conv3d_cuda.cpp:105-149)
//   backward data    SGEMM + col2im_offset + col2im  (deform3d/lib/deform_conv3d_cuda.cpp:186-251)
//   backward weight  deformable_im2col + SGEMM(b=1)  (deform3d/lib/deform_conv3d_cuda.cpp:278-321)
//
// Internal layouts (workspace):
//   x_cl   [N][in volume][C] bf16      channels-last copy of the input: the C/dg channels that share one
//                                      sampling point are contiguous, so one corner fetch is a 16-byte load
//   w_pk   pre-swizzled 128x64 bf16 operand tiles of the weight, GEMM-K ordered (tap, channel)
//   dx_cl  [N][in volume][C] fp32      channels-last input-gradient accumulator (backward data)
//
// Requirements (dcn_precision_supported): fp32 tensors, C/G and C/dg multiples of 8.
#include <stdlib.h>

#include <type_traits>

#include "dcn_internal.h"
#include "dcn_tc_common.cuh"

namespace dcn {

using namespace tc;

namespace {

constexpr int kTileN = 128;            // output positions per tile
constexpr int kTileK = 64;             // bf16 elements per K chunk (one 128-byte swizzled row)
constexpr int kTileBytes = 128 * 128;  // one 128-row operand tile: 16 KB
constexpr int kProducerWarps = 8;
constexpr int kEpilogueWarps = 4;

inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

struct TcDims {
    int KC;         // K chunks per group: ceil(kv*Cg / 64)
    int MT;         // 128-row output-channel tiles per group
    int MB;         // o-blocks per group (each up to 2 m-tiles sharing the sampled operand)
    long long PT;   // position tiles
};

TcDims tc_dims(const Geom& g) {
    TcDims d;
    d.KC = (g.kv * g.Cg + kTileK - 1) / kTileK;
    d.MT = (g.Og + 127) / 128;
    d.MB = (d.MT + 1) / 2;
    d.PT = (g.P + kTileN - 1) / kTileN;
    return d;
}

// ---------------------------------------------------------------------------------------------------
// Sampling of one 16-byte chunk (8 consecutive channels of one tap, one deformable group) at one output
// position, from the channels-last bf16 input.  Returns 8 bf16 packed in 4 words.
// ---------------------------------------------------------------------------------------------------
template <int D, bool DEFORM>
__device__ __forceinline__ uint4 sample_chunk(const Geom& g, const __nv_bfloat16* __restrict__ xcl,
                                              const float* __restrict__ off, const OutPos& op, int tap, int c,
                                              int grp) {
    const uint32_t pix_bytes = (uint32_t)g.C * 2u;
    const void* xn = ptr_mad_u32(xcl + c, (uint32_t)op.n * (uint32_t)g.iv, pix_bytes);
    if (!DEFORM) {
        int idx;
        if (!locate_plain<D>(g, tap, op, idx)) return make_uint4(0, 0, 0, 0);
        return gload(static_cast<const uint4*>(ptr_mad_u32(xn, (uint32_t)idx, pix_bytes)));
    }
    Pt<float, D> s;
    locate<float, D>(g, offset_block<float, D>(g, off, op.n), grp, tap, op, s);
    if (!s.valid) return make_uint4(0, 0, 0, 0);
    int idx[1 << D];
    float cw[1 << D];
    corner_indices<float, D>(g, s, idx);
    corner_weights<float, D>(s, cw);
    uint4 q[1 << D];
#pragma unroll
    for (int e = 0; e < (1 << D); ++e) q[e] = gload(static_cast<const uint4*>(ptr_mad_u32(xn, (uint32_t)idx[e], pix_bytes)));
    float acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.f;
#pragma unroll
    for (int e = 0; e < (1 << D); ++e) {
        const uint32_t wd[4] = {q[e].x, q[e].y, q[e].z, q[e].w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            acc[2 * i] = fmaf(cw[e], bf16_lo(wd[i]), acc[2 * i]);
            acc[2 * i + 1] = fmaf(cw[e], bf16_hi(wd[i]), acc[2 * i + 1]);
        }
    }
    return make_uint4(pack_bf16x2(acc[0], acc[1]), pack_bf16x2(acc[2], acc[3]), pack_bf16x2(acc[4], acc[5]),
                      pack_bf16x2(acc[6], acc[7]));
}

#include "dcn_tc_passes.cuh"
#include "dcn_tc_fwd_direct.cuh"
#include "dcn_tc_sampler.cuh"
#include "dcn_tc_fwd.cuh"

struct FwdWorkspace {
    size_t xcl_off, wpk_off, slices_off, total;       // slices: partial sums of split tiles
    FwdSplit split;
};
// have: bytes there are at most
FwdWorkspace fwd_workspace(const Geom& g, size_t have = SIZE_MAX) {
    const TcDims d = tc_dims(g);
    FwdWorkspace w;
    w.xcl_off = 0;
    w.wpk_off = tc_input_copy_bytes(g);
    w.slices_off = w.wpk_off + align_up((size_t)g.G * d.MT * d.KC * kTileBytes, 256);
    w.split = fwd_split(g, have > w.slices_off ? have - w.slices_off : 0);
    w.total = w.slices_off + align_up((size_t)fwd_slices(w.split) * fwd_slice_bytes(g), 256);
    return w;
}

#include "dcn_tc_wgrad.cuh"
#include "dcn_tc_wgrad2.cuh"
#include "dcn_tc_dgrad.cuh"
#include "dcn_tc_dgrad2.cuh"
#include "dcn_tc_bwd2d.cuh"

struct BwdWeightWorkspace {
    size_t xcl_off, dpk_off, dwpk_off, total;
};
BwdWeightWorkspace bwd_weight_workspace(const Geom& g) {
    const WgDims d = wg_dims(g);
    BwdWeightWorkspace w;
    w.xcl_off = 0;
    w.dpk_off = align_up((size_t)g.N * g.iv * g.C * 2, 256);
    w.dwpk_off = w.dpk_off + align_up((size_t)g.G * d.MT * d.PC * kTileBytes, 256);
    w.total = w.dwpk_off + align_up(dwpk_bytes(g), 256);
    return w;
}

struct BwdDataWorkspace {
    // dwpk, sums (row sums of the dy tiles, for the bias gradient): fused backward only; gath: forward workspace of the
    // transposed convolution
    size_t xcl_off, dpk_off, wpk_off, scale_off, dxcl_off, dxcl_bytes, dwpk_off, sums_off, gath_off, total;
};
size_t gather_dgrad_bytes(const Geom& g);      // 0 unless the problem can take the gather form (any ndim)
BwdDataWorkspace bwd_data_workspace(const Geom& g) {
    const DgDims d = dg_dims(g);
    BwdDataWorkspace w;
    w.xcl_off = 0;
    w.dpk_off = align_up((size_t)g.N * g.iv * g.C * 2, 256);
    w.wpk_off = w.dpk_off + align_up((size_t)g.G * d.MT * d.PC2 * kTileBytes, 256);
    size_t wpk_bytes = (size_t)g.G * d.NB * d.OC * 2 * kTileBytes;
    if (g.Cg % 8 == 0 && b2_wpk_bytes(g) > wpk_bytes) wpk_bytes = b2_wpk_bytes(g);   // slab-wise tiles of dcn_tc_bwd2d.cuh
    w.scale_off = w.wpk_off + align_up(wpk_bytes, 256);
    w.dxcl_off = w.scale_off + 256;                    // two words: bit patterns of max|dy| and max|W|; or the tile counter
    w.dxcl_bytes = align_up((size_t)g.N * g.iv * g.C * 4, 256);
    // the shared-memory-accumulating kernel has no channels-last dX scratch; its sampling-point entries live there
    if (g.Cg % 8 == 0 && b2_points_bytes(g) > w.dxcl_bytes) w.dxcl_bytes = align_up(b2_points_bytes(g), 256);
    w.dwpk_off = w.dxcl_off + w.dxcl_bytes;
    w.sums_off = w.dwpk_off + align_up(dwpk_bytes(g), 256);
    w.gath_off = w.sums_off + align_up((size_t)g.G * d.MT * 128 * d.PC2 * 4, 256);
    w.total = w.gath_off + gather_dgrad_bytes(g);
    return w;
}

// ---------------------------------------------------------------------------------------------------
// Plain convolution, stride 1: the input gradient is itself a plain convolution of dy (taps mirrored, weights
// transposed within each group, padding dil*(k-1) - pad), so it runs on the FORWARD kernel as a gather -- every
// dX element written once, no reductions -- instead of the scatter the deformable operator needs.
// gt: that convolution's geometry (C and O swapped, input and output sizes swapped).
// ---------------------------------------------------------------------------------------------------
bool transposed_geom(const Geom& g, int ndim, Geom& gt) {
    gt = g;
    gt.C = g.O; gt.O = g.C;
    gt.cpg = gt.C; gt.dg = 1; gt.oob = 0;
    gt.iv = g.ov; gt.ov = g.iv;
    for (int d = 0; d < 3; ++d) {
        if (g.stride[d] != 1) return false;
        gt.in[d] = g.out[d]; gt.out[d] = g.in[d];
        gt.pad[d] = g.dil[d] * (g.k[d] - 1) - g.pad[d];
        if (gt.pad[d] < 0) return false;
        if (gt.in[d] + 2 * gt.pad[d] - g.dil[d] * (g.k[d] - 1) != gt.out[d]) return false;
    }
    gt.Cg = g.Og; gt.Og = g.Cg; gt.Kg = gt.Cg * gt.kv;
    gt.P = (long long)gt.N * gt.ov;
    gt.d_ov.init(gt.ov); gt.d_ow.init(gt.out[2]); gt.d_oh.init(gt.out[1]);
    gt.d_Cg.init(gt.Cg); gt.d_cpg.init(gt.cpg);
    (void)ndim;
    return gt.Cg % 8 == 0 && gt.N <= 65535;
}

bool use_gather_dgrad(const Geom& g, int ndim, int deform, Geom& gt) {
    static const bool off = [] { const char* e = getenv("DCN_GATHER_DGRAD"); return e != nullptr && e[0] == '0'; }();
    return !off && !deform && transposed_geom(g, ndim, gt);
}

size_t gather_dgrad_bytes(const Geom& g) {
    Geom gt;
    if (g.dg != 1 || g.cpg != g.C) return 0;                     // deformable problems never take it
    if (!transposed_geom(g, 3, gt)) return 0;
    return align_up(fwd_workspace(gt).total, 256);
}

// The shared-memory-accumulating backward-data kernel is taken whenever it fits (DCN_BWD2D=0 forces the
// global-reduction kernels, for A/B measurements): its dX is a fixed-point sum that does not depend on the order of its
// terms, the other's is added up by reductions in whichever order they arrive.  It is the faster one where its items (one
// sample x eight channels, a whole plane on one SM) fill the SMs, and not where they are few or the planes tiny.  Backward
// data of n x c -> c channels, 3x3, one deformable group, B200, kernel time plane / reductions in us:
//   8 items    1 x 64:  14x14 11 / 18, 28x28 26 / 19, 56x56 84 / 20       32 items   2 x 128: 28x28 27 / 20, 56x56 88 / 35
//   64 items   4 x 128, 56x56 87 / 63; 8 x 64, 56x56 84 / 65              128 items  4 x 256: 14x14 14 / 22, 28x28 31 / 40
//   256 items  8 x 256, 28x28 56 / 54; 32 x 64, 56x56 165 / 209           512 items  16 x 256, 14x14 40 / 39
//   1024 items 32 x 256: 14x14 66 / 52, 56x56 (four groups) 626 / 760
// (about 5 us + 25 ns a position for each wave of items against 15 us + 3.4 ps a sample of C x taps x positions).
bool use_bwd2d(const Geom& g, int ndim, int deform) {
    static const bool off = [] { const char* e = getenv("DCN_BWD2D"); return e != nullptr && e[0] == '0'; }();
    return !off && b2_supported(g, ndim, deform);
}

// The gradient kernels of one convolution and the passes around them: `prologue` adds what has to be done before them
// (it may enqueue a memset), `run` launches them, `epilogue` adds what turns their scratch into the caller's tensors.
// The caller launches the passes, together with those of another convolution where it has one.
struct Backward {
    const Geom& g;
    int ndim, deform;
    bool add;                            // dX and dW accumulate (else they are overwritten)
    const float *off, *w, *dy;
    float *dx, *doff, *dw, *dbias;
    bool dx_cl;                          // dX is stored channels-last (g.cl says so of dy)
    bool dx_partial;                     // dX holds a partial result already (add, for dX alone)
    const __nv_bfloat16* xcl;
    uint8_t* base;
    BwdDataWorkspace l;
    DgDims d;
    bool b2, gather, scatter, tiles, bias_here;
    Geom gt, gk;                         // transposed convolution; with the layout of dX
    FwdPlan plan;                        // of the gather
    FwdWorkspace f;

    Backward(const Geom& g_, int ndim_, int deform_, bool add_, const float* off_, const float* w_, const float* dy_, float* dx_,
             float* doff_, float* dw_, float* dbias_, void* ws)
        : g(g_), ndim(ndim_), deform(deform_), add(add_), off(off_), w(w_), dy(dy_), dx(dx_), doff(deform_ ? doff_ : nullptr),
          dw(dw_), dbias(dbias_), dx_cl(g_.cl != 0), dx_partial(add_), xcl(nullptr), base(static_cast<uint8_t*>(ws)),
          l(bwd_data_workspace(g_)), d(dg_dims(g_)) {
        const bool data = dx != nullptr || doff != nullptr;
        b2 = data && use_bwd2d(g, ndim, deform);
        gather = !b2 && dx != nullptr && use_gather_dgrad(g, ndim, deform, gt);
        scatter = data && !b2 && !gather;
        tiles = b2 || scatter || dw != nullptr;
        bias_here = dbias != nullptr && tiles;
    }
    __nv_bfloat16* own_xcl() const { return reinterpret_cast<__nv_bfloat16*>(base + l.xcl_off); }
    bool needs_x() const { return dw != nullptr || (deform && (b2 || scatter)); }
    unsigned int* scale() const { return reinterpret_cast<unsigned int*>(base + l.scale_off); }
    float* dxcl() const {                // scatter target: a channels-last dX itself, else the scratch
        return dx == nullptr ? nullptr : (dx_cl ? dx : reinterpret_cast<float*>(base + l.dxcl_off));
    }
    float* sums() const { return bias_here ? reinterpret_cast<float*>(base + l.sums_off) : nullptr; }

    // what depends on the weight and the offsets only (`before`), and what needs dy (`with_dy`)
    int before(Passes& p, cudaStream_t st) {
        if (b2) {
            const B2Dims e = b2_dims(g);
            if (cudaMemsetAsync(scale(), 0, 8, st) != cudaSuccess) return -5;
            p.points(g, off, reinterpret_cast<uint4*>(base + l.dxcl_off), e.Wp, e.W2);
            p.weight(g, kTilesSlab, w, base + l.wpk_off, scale() + 1);
        }
        if (scatter) {
            if (dx_cl && dx != nullptr && (reinterpret_cast<uintptr_t>(dx) & 15) != 0) return -7;   // 16-byte reductions
            p.weight(g, kTilesBwd, w, base + l.wpk_off, nullptr, scale());      // (clears the kernel's tile counter)
            if (dx != nullptr && !(dx_cl && dx_partial)) p.zero(dxcl(), (size_t)g.N * g.iv * g.C);
        }
        if (doff != nullptr) p.zero(doff, (size_t)g.N * g.dg * g.kv * ndim * g.ov);
        if (gather) {
            f = fwd_workspace(gt);
            gk = gt;
            gk.cl = dx_cl ? 1 : 0;
            plan = fwd_plan(gk, f.split, ndim, 0, dx, dx_partial);
            if (plan.direct && dx_partial) return -5;
            p.weight(g, kTilesFlip, w, base + l.gath_off + f.wpk_off);
        }
        return 0;
    }
    void with_dy(Passes& p) {
        if (tiles) p.pack_dy(g, dy, base + l.dpk_off, d.MT, d.PC2, b2 ? scale() : nullptr, sums());
        if (gather) p.copy_x(gt, dy, reinterpret_cast<__nv_bfloat16*>(base + l.gath_off + f.xcl_off));
    }
    int run(cudaStream_t st) {
        int r = 0;
        const uint8_t* dpk = base + l.dpk_off;
        if (b2)
            r = launch_tc_bwd2d(g, xcl, reinterpret_cast<uint4*>(base + l.dxcl_off), dpk, base + l.wpk_off, scale(), dx, doff,
                                dx_partial, st);
        if (scatter) {
            if (ndim == 2) r = deform ? launch_tc_dgrad<2, true>(g, xcl, off, dpk, base + l.wpk_off, dxcl(), doff, scale(), st)
                                      : launch_tc_dgrad<2, false>(g, xcl, off, dpk, base + l.wpk_off, dxcl(), doff, scale(), st);
            else r = deform ? launch_tc_dgrad<3, true>(g, xcl, off, dpk, base + l.wpk_off, dxcl(), doff, scale(), st)
                            : launch_tc_dgrad<3, false>(g, xcl, off, dpk, base + l.wpk_off, dxcl(), doff, scale(), st);
        }
        if (r == 0 && gather)            // (a split one is folded behind it, by fold_dx)
            r = launch_tc_forward(gk, plan, ndim, 0, reinterpret_cast<const __nv_bfloat16*>(base + l.gath_off + f.xcl_off), nullptr,
                                  base + l.gath_off + f.wpk_off, nullptr, dx, slices(), st);
        if (r == 0 && dw != nullptr) {   // the weight kernel reads dy tiles with the same layout and stride (PC2 == wg_dims().PC)
            float* dwpk = reinterpret_cast<float*>(base + l.dwpk_off);
            if (ndim == 2) r = deform ? launch_tc_wgrad<2, true>(g, xcl, off, dpk, dwpk, st)
                                      : launch_tc_wgrad<2, false>(g, xcl, off, dpk, dwpk, st);
            else r = deform ? launch_tc_wgrad<3, true>(g, xcl, off, dpk, dwpk, st)
                            : launch_tc_wgrad<3, false>(g, xcl, off, dpk, dwpk, st);
        }
        return r;
    }
    float* slices() const { return reinterpret_cast<float*>(base + l.gath_off + f.slices_off); }
    void fold_dx(Passes& p) const {
        if (scatter && dx != nullptr && !dx_cl) p.fold_dx(g, dxcl(), dx, dx_partial);
        if (gather && plan.folds()) p.fold_y(gk, y_fold(gk, plan, slices(), nullptr, dx));
    }
    void epilogue(Passes& p) const {
        if (dw != nullptr) add_dw_fold(p, g, reinterpret_cast<const float*>(base + l.dwpk_off), dw, add);
        if (bias_here) p.fold_bias(g, sums(), dbias, d.MT, d.PC2);
    }
};

}  // namespace

bool tc_supported(const Geom& g, int ndim, int deform) {
    (void)ndim;
    if (g.Cg % 8 != 0) return false;
    if (deform && g.cpg % 8 != 0) return false;
    if (g.N > 65535) return false;
    return true;
}

size_t tc_workspace_bytes(const Geom& g, int ndim, int pass) {
    (void)ndim;
    if (pass == 0) return fwd_workspace(g).total;
    if (pass == 1) return bwd_data_workspace(g).total;
    return bwd_weight_workspace(g).total;
}

// Kernels a pass enqueues when every gradient of the tensors is wanted (see dcn_launch_count).
int tc_launch_count(const Geom& g, int ndim, int deform, int pass) {
    auto folds = [&](const Geom& f, int df) { return fwd_plan(f, fwd_workspace(f).split, ndim, df, nullptr, false).folds() ? 1 : 0; };
    Geom gt;
    if (pass == 0) return 2 + folds(g, deform);            // prologue, implicit GEMM, (fold of the split tiles)
    if (pass == 1 && use_bwd2d(g, ndim, deform)) return 2; // prologue, GEMM + scatter
    if (pass == 1 && use_gather_dgrad(g, ndim, deform, gt)) return 2 + folds(gt, 0);
    if (pass == 1) return g.cl ? 2 : 3;                    // prologue, GEMM + scatter, (dX transpose)
    if (pass == 2) return 3;                               // prologue, implicit GEMM, dW fold
    return 4;                                              // all gradients: prologue, two GEMMs, epilogue
}

int tc_debug_points(const Geom& g, int ndim, int deform, const float* off, int n, float* coords, int32_t* valid,
                    int32_t* lo, int32_t* hi, void* ws, size_t ws_bytes, cudaStream_t st) {
    if (!b2_supported(g, ndim, deform)) return -3;
    const BwdDataWorkspace l = bwd_data_workspace(g);
    if (ws_bytes < l.total) return -4;
    uint4* pts = reinterpret_cast<uint4*>(static_cast<uint8_t*>(ws) + l.dxcl_off);
    const B2Dims d = b2_dims(g);
    Passes p;
    p.points(g, off, pts, d.Wp, d.W2);
    const int r = p.launch(st, true);
    if (r != 0) return r;
    const long long want = ((long long)g.dg * g.kv * g.ov + 255) / 256;
    const int blocks = (int)(want < 16ll * sm_count() ? want : 16ll * sm_count());
    b2_points_decode_kernel<<<blocks, 256, 0, st>>>(g, pts, n, d.Wp, d.W2, coords, valid, lo, hi);
    return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

size_t tc_input_copy_bytes(const Geom& g) { return align_up((size_t)g.N * g.iv * g.C * 2, 256); }

int tc_forward(const Geom& g, int ndim, int deform, const float* x, const float* off, const float* w,
               const float* bias, float* y, void* xcl_out, void* ws, size_t ws_bytes, cudaStream_t st) {
    const size_t less = xcl_out != nullptr ? tc_input_copy_bytes(g) : 0;      // of the workspace, which starts behind the copy
    const FwdWorkspace l = fwd_workspace(g, ws_bytes + less);
    if (ws_bytes + less < l.total) return -4;
    uint8_t* base = static_cast<uint8_t*>(ws);
    __nv_bfloat16* xcl = static_cast<__nv_bfloat16*>(xcl_out != nullptr ? xcl_out : ws);
    uint8_t* wpk = base + (l.wpk_off - less);
    const FwdPlan plan = fwd_plan(g, l.split, ndim, deform, y, false);
    float* slices = reinterpret_cast<float*>(base + (l.slices_off - less));
    Passes p;
    p.copy_x(g, x, xcl);
    p.weight(g, kTilesFwd, w, wpk);
    int r = p.launch(st, false);
    if (r == 0) r = launch_tc_forward(g, plan, ndim, deform, xcl, off, wpk, bias, y, slices, st);
    return r != 0 ? r : launch_y_fold(g, plan, slices, bias, y, true, st);
}

int tc_backward_data(const Geom& g, int ndim, int deform, const float* x, const float* off, const float* w,
                     const float* dy, float* dx, float* doff, void* ws, size_t ws_bytes, cudaStream_t st) {
    if (ws_bytes < bwd_data_workspace(g).total) return -4;
    Backward b(g, ndim, deform, true, off, w, dy, dx, doff, nullptr, nullptr, ws);     // accumulates into dX
    Passes p;
    int r = b.before(p, st);
    if (r != 0) return r;
    b.with_dy(p);
    if (b.needs_x()) {
        p.copy_x(g, x, b.own_xcl());
        b.xcl = b.own_xcl();
    }
    r = p.launch(st, false);
    if (r == 0) r = b.run(st);
    Passes q;
    b.fold_dx(q);
    return r != 0 ? r : q.launch(st, true);
}

int tc_backward_weight(const Geom& g, int ndim, int deform, const float* x, const float* off, const float* dy,
                       float* dw, void* ws, size_t ws_bytes, cudaStream_t st) {
    const BwdWeightWorkspace l = bwd_weight_workspace(g);
    if (ws_bytes < l.total) return -4;
    uint8_t* base = static_cast<uint8_t*>(ws);
    __nv_bfloat16* xcl = reinterpret_cast<__nv_bfloat16*>(base + l.xcl_off);
    uint8_t* dpk = base + l.dpk_off;
    const WgDims d = wg_dims(g);
    Passes p;
    p.copy_x(g, x, xcl);
    p.pack_dy(g, dy, dpk, d.MT, d.PC, nullptr, nullptr);
    int r = p.launch(st, false);
    if (r != 0) return r;
    float* dwpk = reinterpret_cast<float*>(base + l.dwpk_off);
    if (ndim == 2) r = deform ? launch_tc_wgrad<2, true>(g, xcl, off, dpk, dwpk, st)
                              : launch_tc_wgrad<2, false>(g, xcl, off, dpk, dwpk, st);
    else r = deform ? launch_tc_wgrad<3, true>(g, xcl, off, dpk, dwpk, st)
                    : launch_tc_wgrad<3, false>(g, xcl, off, dpk, dwpk, st);
    if (r != 0) return r;
    Passes q;
    add_dw_fold(q, g, dwpk, dw, true);               // this entry point accumulates into dW
    return q.launch(st, true);
}

// ---------------------------------------------------------------------------------------------------
// Fused backward: all requested gradients in one call.  The channels-last input copy and the packed dy are
// built once and shared by the data and weight kernels (or the input copy is taken over from the forward
// pass), and every output is overwritten, so no caller-side zero fill and no read-modify-write of dx.
// ---------------------------------------------------------------------------------------------------
size_t tc_backward_workspace_bytes(const Geom& g) { return bwd_data_workspace(g).total; }

int tc_backward(const Geom& g, int ndim, int deform, const float* x, const float* off, const float* w,
                const float* dy, const void* xcl_in, float* dx, float* doff, float* dw, float* dbias, bool* bias_done,
                void* ws, size_t ws_bytes, cudaStream_t st) {
    if (ws_bytes < bwd_data_workspace(g).total) return -4;
    Backward b(g, ndim, deform, false, off, w, dy, dx, doff, dw, dbias, ws);
    *bias_done = b.bias_here;
    Passes p;
    int r = b.before(p, st);
    if (r != 0) return r;
    b.with_dy(p);
    b.xcl = static_cast<const __nv_bfloat16*>(xcl_in);
    if (b.xcl == nullptr && b.needs_x()) {
        p.copy_x(g, x, b.own_xcl());
        b.xcl = b.own_xcl();
    }
    r = p.launch(st, false);
    if (r == 0) r = b.run(st);
    if (r != 0) return r;
    Passes q;
    b.fold_dx(q);
    b.epilogue(q);
    return q.launch(st, true);
}

// ---------------------------------------------------------------------------------------------------
// Deformable layer: the plain convolution that produces the offsets (geometry gq: same input, taps, stride and
// padding, dilation 1, one group, dg*kv*D output channels, channel-first output whatever the layout of x)
// followed by the deformable convolution (geometry g) of the same input.  One channels-last bf16 copy of x
// serves both convolutions in the forward pass and all four gradient kernels in the backward pass; the offsets
// are written once and read back while they are still in L2.
// Workspaces: forward  [ forward workspace of g (its start holds the input copy) | forward workspace of gq ]
//             backward [ dOffset | backward workspace of g | backward workspace of gq ]
// ---------------------------------------------------------------------------------------------------
static size_t layer_doff_bytes(const Geom& g, int ndim) {
    return align_up((size_t)g.N * g.dg * g.kv * ndim * g.ov * sizeof(float), 256);
}

size_t tc_layer_workspace_bytes(const Geom& g, const Geom& gq, int ndim, int pass) {
    if (pass == 0) return fwd_workspace(g).total + fwd_workspace(gq).total;
    return layer_doff_bytes(g, ndim) + align_up(bwd_data_workspace(g).total, 256) + align_up(bwd_data_workspace(gq).total, 256);
}

int tc_layer_forward(const Geom& g, const Geom& gq, int ndim, const float* x, const float* w_off, const float* b_off,
                     const float* w, const float* bias, float* offsets, float* y, void* xcl_out, void* ws, size_t ws_bytes,
                     cudaStream_t st) {
    const FwdWorkspace l = fwd_workspace(g), lq = fwd_workspace(gq);
    const size_t less = xcl_out != nullptr ? tc_input_copy_bytes(g) : 0;
    if (ws_bytes + less < l.total + lq.total) return -4;
    uint8_t* base = static_cast<uint8_t*>(ws);
    uint8_t *wpk = base + (l.wpk_off - less), *baseq = base + (l.total - less);
    float *slices = reinterpret_cast<float*>(base + (l.slices_off - less)), *slicesq = reinterpret_cast<float*>(baseq + lq.slices_off);
    __nv_bfloat16* xcl = static_cast<__nv_bfloat16*>(xcl_out != nullptr ? xcl_out : ws);
    const FwdPlan pq = fwd_plan(gq, lq.split, ndim, 0, offsets, false), pl = fwd_plan(g, l.split, ndim, 1, y, false);
    Passes p;
    p.copy_x(g, x, xcl);
    p.weight(gq, kTilesFwd, w_off, baseq + lq.wpk_off);
    p.weight(g, kTilesFwd, w, wpk);
    int r = p.launch(st, false);
    if (r == 0) r = launch_tc_forward(gq, pq, ndim, 0, xcl, nullptr, baseq + lq.wpk_off, b_off, offsets, slicesq, st);
    if (r == 0) r = launch_y_fold(gq, pq, slicesq, b_off, offsets, false, st);
    if (r == 0) r = launch_tc_forward(g, pl, ndim, 1, xcl, offsets, wpk, bias, y, slices, st);
    return r != 0 ? r : launch_y_fold(g, pl, slices, bias, y, true, st);
}

int tc_layer_backward(const Geom& g, const Geom& gq, int ndim, const float* x, const float* offsets, const float* w_off,
                      const float* w, const float* dy, const void* xcl_in, float* dx, float* dw_off, float* db_off, float* dw,
                      float* dbias, float** doff_out, bool* bias_done, bool* bias_off_done, void* ws, size_t ws_bytes,
                      cudaStream_t st) {
    if (ws_bytes < tc_layer_workspace_bytes(g, gq, ndim, 3)) return -4;
    uint8_t* base = static_cast<uint8_t*>(ws);
    float* doff = reinterpret_cast<float*>(base);
    uint8_t* ws_main = base + layer_doff_bytes(g, ndim);
    uint8_t* ws_q = ws_main + align_up(bwd_data_workspace(g).total, 256);
    const bool chain = dx != nullptr || dw_off != nullptr || db_off != nullptr;      // dOffset is needed downstream
    Backward b(g, ndim, 1, false, offsets, w, dy, dx, chain ? doff : nullptr, dw, dbias, ws_main);
    // gradients of the offset-producing convolution given dOffset: its dX is added to the one of the deformable part
    Backward q(gq, ndim, 0, false, nullptr, w_off, doff, dx, nullptr, dw_off, db_off, ws_q);
    q.dx_cl = g.cl != 0;
    q.dx_partial = true;
    *bias_done = b.bias_here;
    *bias_off_done = q.bias_here;
    *doff_out = doff;
    const bool second = dx != nullptr || dw_off != nullptr;
    Passes p;
    b.xcl = static_cast<const __nv_bfloat16*>(xcl_in);
    if (b.xcl == nullptr) {
        p.copy_x(g, x, b.own_xcl());
        b.xcl = b.own_xcl();
    }
    q.xcl = b.xcl;
    int r = b.before(p, st);
    if (r != 0) return r;
    b.with_dy(p);
    if (second) r = q.before(p, st);
    if (r == 0) r = p.launch(st, false);
    if (r == 0) r = b.run(st);
    if (r != 0) return r;
    Passes mid, end;
    b.fold_dx(mid);                      // before anything is added to dX
    if (second) {
        q.with_dy(mid);
        r = mid.launch(st, false);
        if (r == 0) r = q.run(st);
        if (r != 0) return r;
        q.fold_dx(end);
        q.epilogue(end);
    } else {
        r = mid.launch(st, false);
        if (r != 0) return r;
    }
    b.epilogue(end);
    return end.launch(st, true);
}

// ---------------------------------------------------------------------------------------------------
// Forward pass for callers that must not allocate: the scratch (channels-last bf16 copy of the input and
// the packed weight tiles) lives in a fixed array that is part of the library image instead of a
// caller-provided workspace.  Every device that loads the library holds kStaticScratchBytes until the
// process exits.  In host code the array's name is only a stand-in for the symbol; the device address is
// obtained once per device with cudaGetSymbolAddress while that device is current.
// ---------------------------------------------------------------------------------------------------
constexpr size_t kStaticScratchBytes = (size_t)32 << 20;
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

size_t tc_static_scratch_bytes() { return kStaticScratchBytes; }

int tc_forward_static(const Geom& g, int ndim, int deform, const float* x, const float* off, const float* w,
                      const float* bias, float* y, cudaStream_t st) {
    constexpr int kMaxDevices = 64;
    static void* volatile scratch_of_device[kMaxDevices] = {};
    if (fwd_workspace(g, 0).total > kStaticScratchBytes) return -8;      // (without room for a split)
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess) return -5;
    if (dev < 0 || dev >= kMaxDevices) return -8;
    void* ptr = scratch_of_device[dev];
    if (ptr == nullptr) {
        // first call on this device: resolve the array's device address (may load the module)
        if (cudaGetSymbolAddress(&ptr, g_static_scratch) != cudaSuccess || ptr == nullptr) return -5;
        scratch_of_device[dev] = ptr;      // racing first calls resolve the same address
    }
    return tc_forward(g, ndim, deform, x, off, w, bias, y, nullptr, ptr, kStaticScratchBytes, st);
}

// A wait that cannot complete: one thread waits, with a limit of about a millisecond, on a barrier nothing ever
// arrives on.  It must give up, raise the status word and return -- the path every pipeline role of the kernels
// above takes when its bounded wait runs out.  For the test of that path only.
namespace {
__global__ void expire_wait_kernel(long long limit_cycles, int* gave_up) {
    __shared__ uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        fence_barrier_init();
        const bool ok = mbar_wait(&bar, 0, limit_cycles);
        if (gave_up != nullptr) *gave_up = ok ? 0 : 1;
    }
}
}  // namespace

int tc_debug_expire_wait(int* gave_up, cudaStream_t st) {
    expire_wait_kernel<<<1, 32, 0, st>>>(2000000ll, gave_up);
    return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

int tc_check_status(cudaStream_t st) {
    if (cudaStreamSynchronize(st) != cudaSuccess) return -5;
    unsigned int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_tc_status, sizeof(v)) != cudaSuccess) return -5;
    if (v != 0) {
        const unsigned int z = 0;
        cudaMemcpyToSymbol(g_tc_status, &z, sizeof(z));
        return -6;
    }
    return 0;
}

}  // namespace dcn
