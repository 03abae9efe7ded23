// The soft-argmin and the arithmetic of the sweep's backward, shared by the per-step entry points
// (ssg_backward.cu) and those of several references at once (ssg_refine.cu).
#pragma once

#include "ssg_isb_common.cuh"

namespace ssg {

struct SoftParams {
    int ncand;
    float tau;
    float inv_cand[SSG_MAX_CANDIDATES];  // 1 / d_k
};

// q = sum_k w_k / d_k with w = softmax(-F / tau), by an online softmax
struct OnlineSoftmax {
    float m, s, t;
    __device__ __forceinline__ void init() { m = -INFINITY, s = 0.0f, t = 0.0f; }
    __device__ __forceinline__ void push(float x, float invd)
    {
        if (x > m) {
            const float r = expf(m - x);
            s *= r;
            t *= r;
            m = x;
        }
        const float e = expf(x - m);
        s += e;
        t = fmaf(e, invd, t);
    }
};

// d(uv)/d(point) of the double-sphere projection (python/utils.py:75-94), rows u and v
__device__ __forceinline__ void project_jacobian(const float p[3], const TorchCam& k, float ju[3], float jv[3])
{
    const float x = p[0], y = p[1], z = p[2];
    const float d1 = sqrtf(x * x + y * y + z * z);
    const float c = k.xi * d1 + z;
    const float d2 = sqrtf(x * x + y * y + c * c);
    const float nrm = k.alpha * d2 + k.one_minus_alpha * c;
    const float dc[3] = {k.xi * x / d1, k.xi * y / d1, k.xi * z / d1 + 1.0f};
    float dn[3];
    dn[0] = k.alpha * (x + c * dc[0]) / d2 + k.one_minus_alpha * dc[0];
    dn[1] = k.alpha * (y + c * dc[1]) / d2 + k.one_minus_alpha * dc[1];
    dn[2] = k.alpha * (c * dc[2]) / d2 + k.one_minus_alpha * dc[2];
    const float in = 1.0f / nrm, in2 = in * in;
    ju[0] = k.fx * (in - x * dn[0] * in2);
    ju[1] = k.fx * (-x * dn[1] * in2);
    ju[2] = k.fx * (-x * dn[2] * in2);
    jv[0] = k.fy * (-y * dn[0] * in2);
    jv[1] = k.fy * (in - y * dn[1] * in2);
    jv[2] = k.fy * (-y * dn[2] * in2);
}

// The image gradient's fixed-point scale: 2^e with e = 62 - ceil(log2 count) - ceil(log2 m), m the
// largest |dL/dcost| (its float bits) and count a bound on the contributions one texel can receive
// (each at most m x the candidates in magnitude): no sum leaves the int64 range, and a
// contribution is rounded by at most m 2^-(63 - log2 count).  0 when m is 0, inf or NaN.
__device__ __forceinline__ float fixed_scale(uint32_t absmax_bits, double count)
{
    const float m = __uint_as_float(absmax_bits);
    if (!(m > 0.0f) || !(m <= 3.0e38f)) return 0.0f;
    int em, ec;
    frexpf(m, &em);     // m < 2^em
    frexp(count, &ec);  // count < 2^ec
    const int e = max(-120, min(62 - ec - em, 120));
    return ldexpf(1.0f, e);
}

inline SoftParams soft_params(const float* candidates, int ncand, float tau)
{
    SoftParams sp{};
    sp.ncand = ncand;
    sp.tau = tau;
    for (int k = 0; k < ncand; ++k) sp.inv_cand[k] = 1.0f / candidates[k];
    return sp;
}

}  // namespace ssg
