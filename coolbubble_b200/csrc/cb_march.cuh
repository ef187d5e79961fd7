/* cb_march.cuh -- shared-memory accesses of the kernels that march the planes of
 * a 3-D tile with its columns in registers (cb_step3_tb.cu, cb_step3_df.cu). */
#ifndef CB_MARCH_CUH
#define CB_MARCH_CUH

#include <cuda_runtime.h>

#include <cstdint>

namespace cb {
namespace {

/* block-wide barrier (bar.red over all threads), returning whether any
 * thread passed true */
__device__ __forceinline__ bool tb_any(bool x) { return __syncthreads_or(x ? 1 : 0) != 0; }

/* shared-memory accesses by 32-bit shared address */
template <typename V>
__device__ __forceinline__ V lds(uint32_t a);
template <>
__device__ __forceinline__ float lds<float>(uint32_t a) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
}
template <>
__device__ __forceinline__ float2 lds<float2>(uint32_t a) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
    return v;
}
template <>
__device__ __forceinline__ float4 lds<float4>(uint32_t a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}
template <>
__device__ __forceinline__ double lds<double>(uint32_t a) {
    double v;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a));
    return v;
}
template <>
__device__ __forceinline__ double2 lds<double2>(uint32_t a) {
    double2 v;
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ void sts(uint32_t a, float v) {
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void sts(uint32_t a, const float2 &v) {
    asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v.x), "f"(v.y) : "memory");
}
__device__ __forceinline__ void sts(uint32_t a, const float4 &v) {
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
                 : "memory");
}
__device__ __forceinline__ void sts(uint32_t a, double v) {
    asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void sts(uint32_t a, const double2 &v) {
    asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v.x), "d"(v.y) : "memory");
}
/* v = shared value at a where pred != 0 (a predicated load: no branch) */
__device__ __forceinline__ void lds_if(float &v, uint32_t a, uint32_t pred) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p ld.shared.f32 %0, [%1];\n\t}"
                 : "+f"(v)
                 : "r"(a), "r"(pred));
}
__device__ __forceinline__ void lds_if(double &v, uint32_t a, uint32_t pred) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p ld.shared.f64 %0, [%1];\n\t}"
                 : "+d"(v)
                 : "r"(a), "r"(pred));
}

/* the sites of 1, 2 or 4 consecutive positions, by their count */
template <typename T, int N>
struct Part;
template <>
struct Part<float, 1> { using V = float; };
template <>
struct Part<float, 2> { using V = float2; };
template <>
struct Part<float, 4> { using V = float4; };
template <>
struct Part<double, 1> { using V = double; };
template <>
struct Part<double, 2> { using V = double2; };
__device__ __forceinline__ float first(float v) { return v; }
__device__ __forceinline__ float first(const float2 &v) { return v.x; }
__device__ __forceinline__ float first(const float4 &v) { return v.x; }
__device__ __forceinline__ double first(double v) { return v; }
__device__ __forceinline__ double first(const double2 &v) { return v.x; }
__device__ __forceinline__ float last(float v) { return v; }
__device__ __forceinline__ float last(const float2 &v) { return v.y; }
__device__ __forceinline__ float last(const float4 &v) { return v.w; }
__device__ __forceinline__ double last(double v) { return v; }
__device__ __forceinline__ double last(const double2 &v) { return v.y; }

}  // namespace
}  // namespace cb

#endif
