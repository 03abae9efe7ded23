// Projection and sample coordinates of the sweep from packed images (ssg_sweep.cu, ssg_refine.cu): the
// reference's arithmetic, with quotients taken from a reciprocal.
#pragma once

#include "ssg_common.cuh"

namespace ssg {

// a / b rounded to nearest, from r = RN(1 / b): a quotient within an ulp and its exact remainder give
// the rounded quotient (P. W. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34(1), 1990).  Where the quotient or the remainder leaves
// the normal range the result may differ from a / b; here those are coordinates far outside the
// image, or offsets that the following sum absorbs.
__device__ __forceinline__ float div_by_reciprocal(float a, float b, float r)
{
    const float q = fmul(a, r);
    return ffma(ffma(-b, q, a), r, q);
}

// project_torch without the validity flag, its two quotients from one reciprocal
__device__ __forceinline__ void project_packed(const float p[3], const TorchCam& k, float uv[2])
{
    const float d1 = norm3_torch(p[0], p[1], p[2]);
    const float c = fadd(fmul(k.xi, d1), p[2]);
    const float d2 = norm3_torch(p[0], p[1], c);
    const float nrm = fadd(fmul(k.alpha, d2), fmul(k.one_minus_alpha, c));
    const float a = fmul(k.fx, p[0]), b = fmul(k.fy, p[1]);
    float qa, qb;
    if (fabsf(nrm) > 1e-30f && fabsf(nrm) < 1e30f) {
        const float r = __frcp_rn(nrm);
        qa = div_by_reciprocal(a, nrm, r);
        qb = div_by_reciprocal(b, nrm, r);
    } else {
        qa = fdiv(a, nrm);
        qb = fdiv(b, nrm);
    }
    uv[0] = fadd(qa, k.cx);
    uv[1] = fadd(qb, k.cy);
}

__device__ __forceinline__ float packed_sample_coord(float uv, float size, float inv_size)
{
    // inv_size = RN(1 / size): the same quotient for a power of two, where t * inv_size is exact
    const float q = div_by_reciprocal(fadd(uv, 0.5f), size, inv_size);
    return fmul(fsub(fmul(fadd(fsub(fmul(q, 2.0f), 1.0f), 1.0f), size), 1.0f), 0.5f);
}

}  // namespace ssg
