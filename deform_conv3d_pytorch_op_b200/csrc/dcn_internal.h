// Internal interfaces between the C-ABI layer (dcn_api.cu) and the kernel files of libdcn.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>
#include <stdlib.h>

#include <atomic>

#include "dcn_common.cuh"

namespace dcn {

// DCN_PDL=0: plain launches, in order.
inline bool pdl_enabled() {
    static const bool off = [] { const char* e = getenv("DCN_PDL"); return e != nullptr && e[0] == '0'; }();
    return !off;
}

// SMs of the current device, asked for once per device (148 where there is none to ask: sizes are also computed on hosts
// without a GPU).
inline int sm_count() {
    constexpr int kMaxDevices = 64;
    static std::atomic<int> count_of_device[kMaxDevices];
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 148;
    int n = count_of_device[dev];
    if (n == 0) {
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) n = 148;
        count_of_device[dev] = n;              // racing first calls find the same number
    }
    return n;
}

// Launch of a kernel that calls pdl_wait() before it reads or writes global memory (see dcn_common.cuh).
template <typename... P, typename... A>
cudaError_t launch_dependent(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, const A&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, P(args)...);
    return e != cudaSuccess ? e : cudaGetLastError();
}

// EXACT-precision (SIMT) launchers, dcn_simt.cu.  dtype: 0 fp32, 1 fp64.  Return 0 or -5 (launch failure).
int simt_forward(const Geom& g, int dtype, int ndim, int deform, const void* x, const void* off, const void* w,
                 const void* bias, void* y, cudaStream_t st);
int simt_backward_data(const Geom& g, int dtype, int ndim, int deform, const void* x, const void* off,
                       const void* w, const void* dy, void* dx, void* doff, cudaStream_t st);
int simt_backward_weight(const Geom& g, int dtype, int ndim, int deform, const void* x, const void* off,
                         const void* dy, void* dw, cudaStream_t st);
// latency-shaped kernels for very small fp32 deformable problems (dcn_simt_small.cuh)
bool simt_small_supported(const Geom& g, int dtype, int ndim, int deform);
int simt_small_forward(const Geom& g, int ndim, const void* x, const void* off, const void* w, const void* bias,
                       void* y, cudaStream_t st);
int simt_small_backward(const Geom& g, int ndim, const void* x, const void* off, const void* w, const void* dy,
                        void* dx, void* doff, void* dw, void* db, cudaStream_t st);
// fused layer forward for small problems: offsets computed in the kernel (gq: the offset-producing convolution)
bool simt_small_layer_supported(const Geom& g, const Geom& gq, int dtype, int ndim);
int simt_small_layer_forward(const Geom& g, const Geom& gq, int ndim, const void* x, const void* w_off, const void* b_off,
                             const void* w, const void* bias, void* offsets, void* y, cudaStream_t st);
int simt_small_layer_backward(const Geom& g, const Geom& gq, int ndim, const void* x, const void* offsets,
                              const void* w_off, const void* w, const void* dy, void* dx, void* dw_off, void* db_off,
                              void* dw, void* db, cudaStream_t st);
bool simt_backward_both_supported(const Geom& g, int dtype);
int simt_backward_both(const Geom& g, int ndim, int deform, const void* x, const void* off, const void* w,
                       const void* dy, void* dx, void* doff, void* dw, cudaStream_t st);
int bias_grad(const Geom& g, int dtype, const void* dy, void* dbias, cudaStream_t st);
int debug_points(const Geom& g, int dtype, int ndim, const void* off, int n, void* coords, int32_t* valid,
                 int32_t* lo, int32_t* hi, cudaStream_t st);

// EXACT precision over a channels-last copy of the input, dcn_exact.cu (needs a workspace).  pass: 0 forward, 1 backward
// data, 2 backward weight, 3 both; add: dX and dW accumulate instead of being overwritten.
bool exact_supported(const Geom& g, int dtype, int deform);
size_t exact_workspace_bytes(const Geom& g, int dtype, int deform, int pass);
int exact_launch_count(int pass);
int exact_forward(const Geom& g, int dtype, int ndim, int deform, const void* x, const void* off, const void* w,
                  const void* bias, void* y, void* ws, cudaStream_t st);
int exact_backward(const Geom& g, int dtype, int ndim, int deform, int pass, int add, const void* x, const void* off,
                   const void* w, const void* dy, void* dx, void* doff, void* dw, void* db, void* ws, cudaStream_t st);

// BF16 tensor-core (tcgen05) path, dcn_tc.cu.  fp32 tensors only.
bool tc_supported(const Geom& g, int ndim, int deform);
size_t tc_workspace_bytes(const Geom& g, int ndim, int pass);
// xcl_out: where the channels-last copy of x goes, tc_input_copy_bytes() that the workspace then needs less (null: its start)
size_t tc_input_copy_bytes(const Geom& g);
int tc_forward(const Geom& g, int ndim, int deform, const float* x, const float* off, const float* w,
               const float* bias, float* y, void* xcl_out, void* ws, size_t ws_bytes, cudaStream_t st);
int tc_backward_data(const Geom& g, int ndim, int deform, const float* x, const float* off, const float* w,
                     const float* dy, float* dx, float* doff, void* ws, size_t ws_bytes, cudaStream_t st);
int tc_backward_weight(const Geom& g, int ndim, int deform, const float* x, const float* off, const float* dy,
                       float* dw, void* ws, size_t ws_bytes, cudaStream_t st);
size_t tc_backward_workspace_bytes(const Geom& g);
// bias_done: whether dbias came out with the other gradients (it rides on the pass that packs dy)
int tc_backward(const Geom& g, int ndim, int deform, const float* x, const float* off, const float* w,
                const float* dy, const void* xcl_in, float* dx, float* doff, float* dw, float* dbias, bool* bias_done,
                void* ws, size_t ws_bytes, cudaStream_t st);
// deformable layer = offset-producing plain convolution (gq) + deformable convolution (g) of the same input
size_t tc_layer_workspace_bytes(const Geom& g, const Geom& gq, int ndim, int pass);
int tc_layer_forward(const Geom& g, const Geom& gq, int ndim, const float* x, const float* w_off, const float* b_off,
                     const float* w, const float* bias, float* offsets, float* y, void* xcl_out, void* ws, size_t ws_bytes,
                     cudaStream_t st);
int tc_layer_backward(const Geom& g, const Geom& gq, int ndim, const float* x, const float* offsets, const float* w_off,
                      const float* w, const float* dy, const void* xcl_in, float* dx, float* dw_off, float* db_off, float* dw,
                      float* dbias, float** doff_out, bool* bias_done, bool* bias_off_done, void* ws, size_t ws_bytes,
                      cudaStream_t st);
int tc_forward_static(const Geom& g, int ndim, int deform, const float* x, const float* off, const float* w,
                      const float* bias, float* y, cudaStream_t st);
size_t tc_static_scratch_bytes();
int tc_check_status(cudaStream_t st);
int tc_debug_expire_wait(int* gave_up, cudaStream_t st);
int tc_launch_count(const Geom& g, int ndim, int deform, int pass);
int tc_debug_points(const Geom& g, int ndim, int deform, const float* off, int n, float* coords, int32_t* valid,
                    int32_t* lo, int32_t* hi, void* ws, size_t ws_bytes, cudaStream_t st);

}  // namespace dcn
