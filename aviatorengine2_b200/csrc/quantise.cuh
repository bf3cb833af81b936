// quantise.cuh - device construction of a 4-wide node (QNode, fast_trace.cuh)
// from its children's float boxes: the frame, the power-of-two quantum and
// the outward-rounded 8-bit planes.  Shared by the mesh builder
// (fast_build.cu) and the instance-tree refresh (fast.cu).
#pragma once
#include "fast_trace.cuh"

namespace ae {

// Frame of one axis for child boxes spanning [lo, hi]: quantum 2^e and
// origin.  250 quanta cover the span, the origin lies 1/32 quantum below it,
// and the quantum is at least 2^-20 of the coordinates, so that an origin in
// binary32 and the walk's rounding stay small against it.  False when the
// span is beyond the exponent range.
__device__ inline bool axis_frame(float lo, float hi, int &e, float &org) {
    const double need = (double(hi) - double(lo)) / 250.0, mag = fmax(fabs(double(lo)), fabs(double(hi)));
    e = -100;
    if (need > 0.0) e = max(e, ilogb(need) + 1);
    if (mag > 0.0) e = max(e, ilogb(mag) - 20);
    org = __double2float_rd(double(lo) - ldexp(1.0, e) / 32.0);
    return e <= 113 && isfinite(org);
}

// Planes of [a, b] in the frame (org, 2^e), rounded outward with 1/128 of a
// quantum to spare: the walk evaluates a plane to within 2^-8 of a quantum
// (child_hits), so its box always contains [a, b].
__device__ inline bool axis_planes(float org, int e, float a, float b, uint32_t &qa, uint32_t &qb) {
    const double inv = ldexp(1.0, -e);
    const double la = floor((double(a) - double(org)) * inv - 0.0078125);
    const double lb = ceil((double(b) - double(org)) * inv + 0.0078125);
    qa = uint32_t(fmin(fmax(la, 0.0), 255.0));
    qb = uint32_t(fmin(fmax(lb, 0.0), 255.0));
    return la >= 0.0 && lb <= 255.0;
}

// Fills a node's frame and planes from the boxes of its first `n` children
// (min, max; valid[k] false: the slot never hits).  child[] is untouched.
// False when a box cannot be quantised conservatively (every slot is then
// unused).
__device__ inline bool quantise_node(QNode &q, int n, const float (*box)[6], const bool *valid, float *u) {
    for (int a = 0; a < 3; a++) { u[a] = __int_as_float(0x7f800000); u[3 + a] = -__int_as_float(0x7f800000); }
    bool any = false, good = true;
    for (int k = 0; k < n; k++) {
        if (!valid[k]) continue;
        any = true;
        for (int a = 0; a < 3; a++) { u[a] = fminf(u[a], box[k][a]); u[3 + a] = fmaxf(u[3 + a], box[k][3 + a]); }
    }
    int e[3] = {0, 0, 0};
    float org[3] = {0.0f, 0.0f, 0.0f};
    for (int a = 0; a < 3 && any; a++) good = axis_frame(u[a], u[3 + a], e[a], org[a]) && good;
    uint32_t pl[4][6];
    for (int k = 0; k < n; k++)
        for (int a = 0; a < 3; a++)
            if (valid[k] && good) good = axis_planes(org[a], e[a], box[k][a], box[k][3 + a], pl[k][a], pl[k][3 + a]) && good;
    q.ox = org[0]; q.oy = org[1]; q.oz = org[2];
    q.scale = uint32_t(n) << 24;
    if (any && good)
        for (int a = 0; a < 3; a++) q.scale |= uint32_t(e[a] + 141) << (8 * a);
    for (int k = 0; k < 4; k++) {
        const bool use = k < n && good && valid[k];
        q.plane[k] = use ? make_uint2(pl[k][0] | pl[k][1] << 8 | pl[k][2] << 16 | pl[k][3] << 24,
                                      pl[k][4] | pl[k][5] << 8 | kPlaneTail)
                         : make_uint2(0u, kPlaneUnused);
    }
    return good;
}

}  // namespace ae
