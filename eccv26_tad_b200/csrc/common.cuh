// Shared host/device helpers of libsvtad.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdarg>
#include <cstdio>

#include "../../include/svtad.h"

namespace svtad {

// ---- host-side error reporting (thread-local text behind svtad_last_error_string) ----
int set_error(int code, const char* fmt, ...);
#define SV_CHECK_ARG(cond, ...) \
    do { if (!(cond)) return ::svtad::set_error(SVTAD_ERR_ARG, __VA_ARGS__); } while (0)
#define SV_CUDA(expr)                                                                         \
    do {                                                                                      \
        cudaError_t e__ = (expr);                                                             \
        if (e__ != cudaSuccess)                                                               \
            return ::svtad::set_error(SVTAD_ERR_CUDA, "%s failed: %s", #expr,                 \
                                      cudaGetErrorString(e__));                               \
    } while (0)
#define SV_LAUNCH_CHECK(name)                                                                 \
    do {                                                                                      \
        cudaError_t e__ = cudaGetLastError();                                                 \
        if (e__ != cudaSuccess)                                                               \
            return ::svtad::set_error(SVTAD_ERR_CUDA, "launch of %s failed: %s", name,        \
                                      cudaGetErrorString(e__));                               \
    } while (0)

inline size_t dtype_size(int dtype) { return dtype == SVTAD_F32 ? 4 : 2; }
inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

// ---- launchers implemented in the other translation units ----
struct ConvArgs {
    const void* a;        // gathered operand: x (fwd) or gy (dgrad)
    const int32_t* nbr;
    const void* w;
    const void* bias;     // fwd only, may be null
    void* out;
    int64_t n;
    int cin, cout, kk, tpb, dtype;
    const void* plan = nullptr;   // the table's work plan, if the call brings one
};

// CUDA-core kernels (conv_simt.cu)
int simt_fwd(const ConvArgs& p, cudaStream_t s);
int simt_dgrad_gather(const ConvArgs& p, const int32_t* status, cudaStream_t s);
int simt_dgrad_scatter(const ConvArgs& p, const int32_t* status, float* ws, cudaStream_t s);
int simt_wgrad(const void* gy, const void* x, const int32_t* nbr, void* gw, void* gb, int64_t n,
               int cin, int cout, int kk, int tpb, int dtype, int grad_dtype, void* ws, size_t ws_bytes,
               cudaStream_t s);
size_t simt_wgrad_ws_bytes(int64_t n, int cin, int cout, int kk, int dtype);

// fp32 kernels over compacted pairs (conv_f32.cu); channel counts are multiples of 4
bool f32_supported(int cin, int cout, int kk, int dtype);
int f32_fwd(const ConvArgs& p, cudaStream_t s);
int f32_dgrad(const ConvArgs& p, const int32_t* status, cudaStream_t s);
int f32_wgrad(const void* gy, const void* x, const int32_t* nbr, void* gw, void* gb, int64_t n, int cin, int cout, int kk,
              int tpb, void* ws, size_t ws_bytes, cudaStream_t s);
size_t f32_wgrad_ws_bytes(int64_t n, int cin, int cout, int kk);
int forced_path();              // SVTAD_FORCE_PATH: 0 = automatic, 1 = CUDA-core kernels, 2 = tensor-core kernels

// fp32 kernels on the tensor cores (conv_f32_tc.cu)
bool f32_tc_wanted(int op, int64_t n, int cin, int cout, int kk);
int f32_tc_fwd(const ConvArgs& p, cudaStream_t s);
int f32_tc_dgrad(const ConvArgs& p, const int32_t* status, cudaStream_t s);
int f32_tc_wgrad(const void* gy, const void* x, const int32_t* nbr, void* gw, void* gb, int64_t n, int cin, int cout, int kk,
                 int tpb, float* ws_w, float* ws_b, int limit, cudaStream_t s);

// tcgen05 kernels (conv_tc.cu)
bool tc_supported(int op, int64_t n, int cin, int cout, int kk, int dtype);
int tc_fwd(const ConvArgs& p, cudaStream_t s);
int tc_dgrad(const ConvArgs& p, const int32_t* status, cudaStream_t s);
// fit: take no more token splits than the workspace holds the partials of (at least one)
int tc_wgrad(const void* gy, const void* x, const int32_t* nbr, void* gw, void* gb, int64_t n,
             int cin, int cout, int kk, int tpb, int dtype, int grad_dtype, void* ws, size_t ws_bytes, bool fit,
             cudaStream_t s);
size_t tc_wgrad_ws_bytes(int64_t n, int cin, int cout, int kk);
size_t tc_wgrad_partials(long splits, bool with_bias, int cin, int cout, int kk);     // of that many token splits
// svtad_conv_wgrad in a workspace of a given size: the smallest it can do with, and the call
size_t wgrad_least_ws_bytes(int64_t n, int cin, int cout, int kk, int dtype, bool with_bias);
int conv_wgrad_fit(const void* gy, const void* x, const int32_t* nbr, void* gw, void* gb, int64_t n, int cin, int cout, int kk,
                   int tpb, int dtype, void* ws, size_t ws_bytes, cudaStream_t s);
int tc_read_error(int32_t* code_out);
int tc_set_share(int n);
int tc_get_share();
int tc_num_sms();               // of the current device
int tc_ensure_smem(const void* kern, size_t bytes);
int tc_set_share_floor(int n);

// the single-CTA tensor-core kernels behind tc_* (conv_tc_hybrid.cu)
#define SV_DECLARE_TC_FAMILY(prefix)                                                                        \
    int prefix##_fwd(const ConvArgs& p, cudaStream_t s);                                                    \
    int prefix##_dgrad(const ConvArgs& p, const int32_t* status, cudaStream_t s);                           \
    int prefix##_wgrad(const void* gy, const void* x, const int32_t* nbr, void* gw, void* gb, int64_t n,    \
                       int cin, int cout, int kk, int tpb, int dtype, int grad_dtype, void* ws,             \
                       size_t ws_bytes, bool fit, cudaStream_t s);
SV_DECLARE_TC_FAMILY(hybrid)
int hybrid_split(int cn, long m_tiles, int steps, bool dgrad, int& G);    // column block and size of clusters that share a tile's K steps, or 0
// forward / dgrad on CTA pairs (conv_tc_pair.cu)
int pair_fwd(const ConvArgs& p, cudaStream_t s);
int pair_dgrad(const ConvArgs& p, const int32_t* status, cudaStream_t s);

// weight gradient over the pairs of a plan (conv_tc_pairs.cu)
bool pairs_wgrad_wanted(int cin, int kk);
size_t pairs_wgrad_ws_bytes(int cin, int cout);
int pairs_wgrad(const void* gy, const void* x, const void* plan, void* gw, void* gb, int64_t n, int cin, int cout, int kk,
                int dtype, int grad_dtype, void* ws, size_t ws_bytes, cudaStream_t s);

#ifdef __CUDACC__
// ---- launches that may begin before the kernel in front of them has ended ----
// The CTAs of such a kernel are placed while the predecessor's last ones still run and set themselves up; pdl_wait()
// holds them until everything the predecessor wrote can be seen, so it comes before a kernel's first access to global
// memory, reads and writes alike, and before any return.  pdl_trigger() lets the successor's CTAs come in turn.  Back
// to back this hides a launch's 2 us or so (16-bit forward of 2868 rows, C=256: 14.3 -> 12.3 us a call; three pruning
// rounds of two clips: 49 -> 42.5 us).  Kernels of many small CTAs do without the trigger: the successor's, resident early,
// cost the per-slice table builder 1 to 5 of 8 to 12 us; its launch alone, under the predecessor's tail, gains 1.3 us, since
// kernels of a stream otherwise start 2 us apart at the least.  No early start where the caller says that kernels of
// several streams share the GPU: a CTA that waits here holds an SM that another stream's kernel could work on (forward
// and backward of three layers on their streams, hints 3 / 2 / 2: 91 us a step with early starts, 82 without).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <bool PDL, typename... KArgs, typename... Args>
inline cudaError_t launch_as(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, int cluster, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    if (cluster > 1) {
        cudaLaunchAttribute& a = attr[cfg.numAttrs++];
        a.id = cudaLaunchAttributeClusterDimension;
        a.val.clusterDim.x = cluster;
        a.val.clusterDim.y = 1;
        a.val.clusterDim.z = 1;
    }
    if (PDL && tc_get_share() == 1) {
        cudaLaunchAttribute& a = attr[cfg.numAttrs++];
        a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        a.val.programmaticStreamSerializationAllowed = 1;
    }
    cfg.attrs = attr;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, int cluster, Args... args) {
    return launch_as<true>(kern, grid, block, smem, s, cluster, args...);
}
template <typename... KArgs, typename... Args>
inline cudaError_t launch_plain(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, int cluster, Args... args) {
    return launch_as<false>(kern, grid, block, smem, s, cluster, args...);
}

// ---- device helpers ----
template <typename T> struct Cvt;
template <> struct Cvt<float> {
    static __device__ __forceinline__ float4 load4(const float* p) {
        return __ldg(reinterpret_cast<const float4*>(p));
    }
    static __device__ __forceinline__ float load1(const float* p) { return __ldg(p); }
    static __device__ __forceinline__ void store4(float* p, float4 v) {
        *reinterpret_cast<float4*>(p) = v;
    }
    static __device__ __forceinline__ void store1(float* p, float v) { *p = v; }
    static __device__ __forceinline__ float value(float v) { return v; }
};
template <> struct Cvt<__nv_bfloat16> {
    static __device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
        uint2 r = __ldg(reinterpret_cast<const uint2*>(p));
        float4 v;
        v.x = __uint_as_float(r.x << 16);
        v.y = __uint_as_float(r.x & 0xffff0000u);
        v.z = __uint_as_float(r.y << 16);
        v.w = __uint_as_float(r.y & 0xffff0000u);
        return v;
    }
    static __device__ __forceinline__ float load1(const __nv_bfloat16* p) {
        return __bfloat162float(*p);
    }
    static __device__ __forceinline__ void store4(__nv_bfloat16* p, float4 v) {
        __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y);
        __nv_bfloat162 b = __floats2bfloat162_rn(v.z, v.w);
        uint2 r;
        r.x = *reinterpret_cast<uint32_t*>(&a);
        r.y = *reinterpret_cast<uint32_t*>(&b);
        *reinterpret_cast<uint2*>(p) = r;
    }
    static __device__ __forceinline__ void store1(__nv_bfloat16* p, float v) {
        *p = __float2bfloat16_rn(v);
    }
    static __device__ __forceinline__ float value(__nv_bfloat16 v) { return __bfloat162float(v); }
};
template <> struct Cvt<__half> {
    static __device__ __forceinline__ float4 load4(const __half* p) {
        uint2 r = __ldg(reinterpret_cast<const uint2*>(p));
        __half2 a = *reinterpret_cast<__half2*>(&r.x);
        __half2 b = *reinterpret_cast<__half2*>(&r.y);
        float2 fa = __half22float2(a), fb = __half22float2(b);
        return make_float4(fa.x, fa.y, fb.x, fb.y);
    }
    static __device__ __forceinline__ float load1(const __half* p) { return __half2float(*p); }
    static __device__ __forceinline__ void store4(__half* p, float4 v) {
        __half2 a = __floats2half2_rn(v.x, v.y);
        __half2 b = __floats2half2_rn(v.z, v.w);
        uint2 r;
        r.x = *reinterpret_cast<uint32_t*>(&a);
        r.y = *reinterpret_cast<uint32_t*>(&b);
        *reinterpret_cast<uint2*>(p) = r;
    }
    static __device__ __forceinline__ void store1(__half* p, float v) { *p = __float2half_rn(v); }
    static __device__ __forceinline__ float value(__half v) { return __half2float(v); }
};
#endif  // __CUDACC__

}  // namespace svtad
