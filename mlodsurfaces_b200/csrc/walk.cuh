// walk.cuh -- device helpers shared by the tree walks (project.cu, packet.cu,
// gather.cu).
#pragma once

#include "mlods_internal.cuh"

namespace mlods
{
constexpr float kPiRef = 3.14159265f;  // the reference's literal (Fastapss.cu:93)

// Sphere fit + projection of the query (frame origin) in double; mirrors
// Fastapss.cu:354-395 (GPU rule) and CPUUtils.cpp:744-781 (CPU rule).
// Returns false when the result is NaN (caller keeps the input, normal 0).
__device__ __forceinline__ bool fit_sphere(const float* s, double step_max, bool gpu_rule, double x[3], float nrm[3])
{
    const double Sw = s[0];
    const double Sn[3] = {s[1], s[2], s[3]};
    const double Sp[3] = {s[4], s[5], s[6]};
    const double Spn = s[7], Spp = s[8];
    const double u4 = 0.5 * (Spn - (Sp[0] * Sn[0] + Sp[1] * Sn[1] + Sp[2] * Sn[2]) / Sw) /
                      (Spp - (Sp[0] * Sp[0] + Sp[1] * Sp[1] + Sp[2] * Sp[2]) / Sw);
    double u123[3];
    for (int a = 0; a < 3; ++a) u123[a] = (Sn[a] - 2.0 * u4 * Sp[a]) / Sw;
    const double u0 = -((Sp[0] * u123[0] + Sp[1] * u123[1] + Sp[2] * u123[2]) + u4 * Spp) / Sw;
    const double thr = gpu_rule ? 1e-6 : 1e-12;
    double nv[3];
    if (fabs(u4) < thr) {
        const double m[3] = {-u123[0], -u123[1], -u123[2]};
        const double lambda = u0 / (m[0] * m[0] + m[1] * m[1] + m[2] * m[2]);
        for (int a = 0; a < 3; ++a) x[a] = lambda * m[a];
        for (int a = 0; a < 3; ++a) nv[a] = Sn[a];
    } else {
        double c[3];
        for (int a = 0; a < 3; ++a) c[a] = u123[a] / (-2.0 * u4);
        const double r2 = c[0] * c[0] + c[1] * c[1] + c[2] * c[2] - u0 / u4;
        const double rad = sqrt(r2 > 0.0 ? r2 : 0.0);
        double pc[3] = {-c[0], -c[1], -c[2]};
        const double pl = sqrt(pc[0] * pc[0] + pc[1] * pc[1] + pc[2] * pc[2]);
        if (pl != 0.0 || !gpu_rule)
            for (int a = 0; a < 3; ++a) pc[a] /= pl;
        else
            pc[0] = pc[1] = pc[2] = 0.0;
        for (int a = 0; a < 3; ++a) x[a] = c[a] + rad * pc[a];
        for (int a = 0; a < 3; ++a) nv[a] = u123[a] + 2.0 * u4 * x[a];
    }
    const double nl = sqrt(nv[0] * nv[0] + nv[1] * nv[1] + nv[2] * nv[2]);
    if (nl != 0.0 || !gpu_rule)
        for (int a = 0; a < 3; ++a) nv[a] /= nl;
    else
        nv[0] = nv[1] = nv[2] = 0.0;
    if (isnan(x[0]) || isnan(x[1]) || isnan(x[2])) return false;
    const double step = sqrt(x[0] * x[0] + x[1] * x[1] + x[2] * x[2]);
    if (step > step_max)
        for (int a = 0; a < 3; ++a) x[a] *= step_max / step;
    for (int a = 0; a < 3; ++a) nrm[a] = float(nv[a]);
    return true;
}

// Weight with the number of multi-Gaussian terms fixed at compile time
// (NSIG > 0) or read at run time (NSIG == 0); KTYPE < 0 reads the kernel type
// at run time too (uniform across a warp).
template <int KTYPE, int NSIG>
__device__ __forceinline__ float weight_n(const KernelConsts& kc, float d2)
{
    if (KTYPE < 0) {
        if (kc.type == MLODS_GAUSSIAN) return kernel_weight<MLODS_GAUSSIAN>(kc, d2);
        if (kc.type == MLODS_SINGULAR) return kernel_weight<MLODS_SINGULAR>(kc, d2);
        return kernel_weight<MLODS_GAUSSIAN_MULTIPLE>(kc, d2);
    }
    if (KTYPE == MLODS_GAUSSIAN_MULTIPLE && NSIG > 0) {
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < NSIG; ++i) s = fmaf(exp2f(d2 * kc.ms_scale[i]), kc.ms_w[i], s);
        return s;
    }
    return kernel_weight<KTYPE>(kc, d2);
}

__device__ __forceinline__ float rcp_fast(float v)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}

// A value of each of the lane's two nodes.  Plain scalar arithmetic: packing the
// nodes' loaded components into register pairs costs the moves that the packed
// instructions save (226 against 232 ms on the precision workload).
struct Two {
    float x, y;
};
__device__ __forceinline__ Two two(float x, float y) { return Two{x, y}; }
__device__ __forceinline__ Two operator+(Two a, Two b) { return Two{a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ Two operator-(Two a, float b) { return Two{a.x - b, a.y - b}; }
__device__ __forceinline__ Two operator-(Two a, Two b) { return Two{a.x - b.x, a.y - b.y}; }
__device__ __forceinline__ Two operator*(Two a, Two b) { return Two{a.x * b.x, a.y * b.y}; }
__device__ __forceinline__ Two operator*(float a, Two b) { return Two{a * b.x, a * b.y}; }
__device__ __forceinline__ Two fma2(Two a, Two b, Two c) { return Two{fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y)}; }

// v + the value o lanes below, where there is one
__device__ __forceinline__ int add_from_below(int v, int o)
{
    int r;
    asm volatile(
        "{\n .reg .pred p;\n .reg .s32 t;\n shfl.sync.up.b32 t|p, %1, %2, 0, 0xffffffff;\n"
        " @p add.s32 t, t, %1;\n @!p mov.s32 t, %1;\n mov.s32 %0, t;\n}"
        : "=r"(r)
        : "r"(v), "r"(o));
    return r;
}

}  // namespace mlods
