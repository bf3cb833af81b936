// quantise.cuh - device construction of a 4-wide node (QNode, fast_trace.cuh)
// from its children's float boxes: the frame, the power-of-two quantum and
// the outward-rounded 8-bit planes.  Shared by the mesh builder
// (fast_build.cu) and the instance-tree refresh (fast.cu).
#pragma once
#include "fast_trace.cuh"

namespace ae {

// V(q) of QNode.
__device__ inline double plane_value(int q) { return q < 128 ? 2.0 + q / 64.0 : 4.0 + (q - 128) / 32.0; }

// Room between a box and its decoded planes, in units of the scale.  The walks
// compute a plane's distance as V(q) 2^e / d + (o - p) / d, whose second term
// is rounded twice (2^-24 each) and reaches 8 scales beyond the distance
// itself: 2^-20 of the scale, where the relative widening (kExitGrow) covers
// only the distance's share.  Twice that keeps a ray that starts on a box's
// face from missing it: without the room, rays from 0.001 before the floor of a
// mesh 100 units wide missed it in 84,042 of 400,000 cases whose distance
// rounds to about tnear.  A plane step is 2^-6, so boxes do not grow otherwise.
constexpr double kPlaneRoom = 1.9073486328125e-06;  // 2^-19

// Frame of one axis for child boxes spanning [lo, hi]: the smallest scale 2^e
// whose planes reach from lo to hi, and an origin with plane 0 at or below lo,
// both with kPlaneRoom.  The scale is at least 2^-20 of the coordinates.  False
// when the span is beyond the exponent range.
__device__ inline bool axis_frame(float lo, float hi, int &e, float &org) {
    const double need = (double(hi) - double(lo)) / 5.96875, mag = fmax(fabs(double(lo)), fabs(double(hi)));
    e = -100;
    if (need > 0.0) e = max(e, ilogb(need));
    if (mag > 0.0) e = max(e, ilogb(mag) - 20);
    for (;; e++) {
        org = __double2float_rd(double(lo) - (2.0 + kPlaneRoom) * ldexp(1.0, e));
        if (e > 120 || !isfinite(org)) return false;
        if (double(org) + (plane_value(255) - kPlaneRoom) * ldexp(1.0, e) >= double(hi)) return true;
    }
}

// Planes of [a, b] in the frame (org, 2^e): the nearest ones that leave
// kPlaneRoom outside it.
__device__ inline bool axis_planes(float org, int e, float a, float b, uint32_t &qa, uint32_t &qb) {
    const double s = ldexp(1.0, e), va = (double(a) - double(org)) / s - kPlaneRoom,
                 vb = (double(b) - double(org)) / s + kPlaneRoom;
    int lo = int(floor(va < 4.0 ? (va - 2.0) * 64.0 : 128.0 + (va - 4.0) * 32.0));
    int hi = int(ceil(vb <= 4.0 ? (vb - 2.0) * 64.0 : 128.0 + (vb - 4.0) * 32.0));
    lo = min(max(lo, 0), 255);
    hi = min(max(hi, 0), 255);
    qa = uint32_t(lo);
    qb = uint32_t(hi);
    return plane_value(lo) <= va && plane_value(hi) >= vb;
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
    q.scale = 0u;
    if (any && good)
        for (int a = 0; a < 3; a++) q.scale |= uint32_t(e[a] + 127) << (8 * a);
    for (int k = 0; k < 4; k++) {
        const bool use = k < n && good && valid[k];
        q.plane[k] = use ? make_uint2(pl[k][0] | pl[k][1] << 8 | pl[k][2] << 16 | pl[k][3] << 24,
                                      pl[k][4] | pl[k][5] << 8 | kPlaneTail)
                         : make_uint2(0u, kPlaneUnused);
    }
    return good;
}

}  // namespace ae
