// detect.cuh - separately rounded detection predicates shared by the BVH and step kernels.
//
//   segment AABB        collision.cu:10-37   (buildAABBs, velocity radius included)
//   narrow-phase keep   collision.cu:39-92   (buildCollisionList: glue/neighbour exemptions,
//                                             closest points, d^2 < r^2)
//   step-size limit     collision.cu:121-159 (recomputeStepLimitKernel)
//
// The pair test is always evaluated with the lower segment index as segment A, so both
// segments of a pair reach the same decision and every contact list is symmetric.
#pragma once
#include "engine.cuh"

namespace yb {

template <typename R>
struct Box {
    R mn[3], mx[3];
};

// Padded AABB of segment k (k has hasNext).  reach: the larger predicted displacement of its
// endpoints (0 without the velocity radius), its share of a pair's filter distance.
template <typename R>
__device__ __forceinline__ Box<R> segment_box(const Dev<R>& d, int k, const SceneParams<R>& sp, R& reach) {
    typedef Ex<R> E;
    const V4<R> p0 = d.pos[k];
    const V4<R> p1 = d.pos[k + 1];
    R pad = sp.sdr;
    reach = R(0);
    if (sp.useVelRadius) {
        const D2<R> dk = d.dx[0][k];
        const R l0 = xlen2(xyz(dk.a));
        const R l1 = xlen2(xyz(dk.b));
        reach = E::sqrt(ymax(l0, l1));
        pad = E::add(pad, reach);
    }
    Box<R> b;
    b.mn[0] = E::sub(ymin(p0.x, p1.x), pad);
    b.mn[1] = E::sub(ymin(p0.y, p1.y), pad);
    b.mn[2] = E::sub(ymin(p0.z, p1.z), pad);
    b.mx[0] = E::add(ymax(p0.x, p1.x), pad);
    b.mx[1] = E::add(ymax(p0.y, p1.y), pad);
    b.mx[2] = E::add(ymax(p0.z, p1.z), pad);
    return b;
}

// The same box in single precision, rounded outwards (exact in the FP32 build); one that is not
// a number is empty.  lo.w holds an id (-1: no segment), hi.w is free.  The empty box meets a box that is
// unbounded on every axis (a segment whose predicted displacement overflows has one), so a test against a
// box that may be a placeholder looks at the id too.
__device__ __forceinline__ float box_down(float x) { return x; }
__device__ __forceinline__ float box_up(float x) { return x; }
__device__ __forceinline__ float box_down(double x) { return __double2float_rd(x); }
__device__ __forceinline__ float box_up(double x) { return __double2float_ru(x); }
__device__ __forceinline__ float4 empty_lo() { return make_float4(INFINITY, INFINITY, INFINITY, __int_as_float(-1)); }
__device__ __forceinline__ float4 empty_hi() { return make_float4(-INFINITY, -INFINITY, -INFINITY, 0.f); }

__device__ __forceinline__ bool boxes_meet(const float4& alo, const float4& ahi, const float4& blo, const float4& bhi) {
    return alo.x <= bhi.x && blo.x <= ahi.x && alo.y <= bhi.y && blo.y <= ahi.y && alo.z <= bhi.z && blo.z <= ahi.z;
}
template <typename R>
__device__ __forceinline__ void float_box(const Box<R>& b, float4& lo, float4& hi) {
    lo = make_float4(box_down(b.mn[0]), box_down(b.mn[1]), box_down(b.mn[2]), 0.f);
    hi = make_float4(box_up(b.mx[0]), box_up(b.mx[1]), box_up(b.mx[2]), 0.f);
    if (!(lo.x <= hi.x && lo.y <= hi.y && lo.z <= hi.z)) {
        lo = empty_lo();
        hi = empty_hi();
    }
}

// The same box rounded to nearest, for the union that bounds() reports; a test of it widens it by one
// float on each side (in the FP32 build it is exact and stays).
template <typename R>
__device__ __forceinline__ void nearest_box(const Box<R>& b, float4& lo, float4& hi) {
    lo = make_float4((float)b.mn[0], (float)b.mn[1], (float)b.mn[2], 0.f);
    hi = make_float4((float)b.mx[0], (float)b.mx[1], (float)b.mx[2], 0.f);
    if (!(lo.x <= hi.x && lo.y <= hi.y && lo.z <= hi.z)) {
        lo = empty_lo();
        hi = empty_hi();
    }
}
template <typename R>
__device__ __forceinline__ void widen_box(float4& lo, float4& hi) {
    if constexpr (sizeof(R) == 8) {
        const float tiny = __uint_as_float(1u);  // the smallest float: the directed sum is the next one
        lo.x = __fadd_rd(lo.x, -tiny); lo.y = __fadd_rd(lo.y, -tiny); lo.z = __fadd_rd(lo.z, -tiny);
        hi.x = __fadd_ru(hi.x, tiny); hi.y = __fadd_ru(hi.y, tiny); hi.z = __fadd_ru(hi.z, tiny);
    }
}

// Narrow-phase decision for segments x < y (both with hasNext, same scene): not joined by a
// connection, not neighbours on a yarn, and closer than the filter distance, to which each
// segment adds its reach.
template <typename R>
__device__ __forceinline__ bool pair_joined(const Dev<R>& d, int x, int y) {
    const int c0 = d.vp[x].cid;
    const int c1 = d.vp[x + 1].cid;
    return c0 == y || c1 == y || c0 == y + 1 || c1 == y + 1;
}

template <typename R>
__device__ __forceinline__ R pair_distance2(const Dev<R>& d, int x, int y) {
    const V3<R> a0 = xyz(d.pos[x]);
    const V3<R> a1 = xsub(xyz(d.pos[x + 1]), a0);
    const V3<R> b0 = xsub(xyz(d.pos[y]), a0);
    const V3<R> b1 = xsub(xyz(d.pos[y + 1]), a0);
    const UVT<R> uv = closest_uv_exact(a1, b0, b1);
    const V3<R> nrm = xsub(xscale(uv.u, a1), xmix(b0, b1, uv.v));
    return xlen2(nrm);
}

template <typename R>
__device__ __forceinline__ bool pair_within(R d2, R reachX, R reachY, const SceneParams<R>& sp) {
    typedef Ex<R> E;
    R r = E::mul(R(2), sp.sdr);
    if (sp.useVelRadius) {
        r = E::add(r, reachX);
        r = E::add(r, reachY);
    }
    return d2 < E::mul(r, r);
}

template <typename R>
__device__ __forceinline__ R segment_reach(const Dev<R>& d, int k) {
    const D2<R> dk = d.dx[0][k];
    return Ex<R>::sqrt(ymax(xlen2(xyz(dk.a)), xlen2(xyz(dk.b))));
}

template <typename R>
__device__ __forceinline__ bool pair_keep(const Dev<R>& d, int x, int y, const SceneParams<R>& sp) {
    if (pair_joined(d, x, y) || y - x <= 2) return false;
    const R d2 = pair_distance2(d, x, y);
    const bool vr = sp.useVelRadius != 0;
    return pair_within(d2, vr ? segment_reach(d, x) : R(0), vr ? segment_reach(d, y) : R(0), sp);
}

// Appends y to x's contact list.  The count keeps growing past MAX_COLS so that the list
// kernel can report the overflow (collision.cu:80-90).
template <typename R>
__device__ __forceinline__ void list_append(const Dev<R>& d, int x, int y) {
    const int pos = atomicAdd(&d.numCols[x], 1);
    if (pos < MAX_COLS) d.cols[col_at(x, pos)] = y;
}

// Step-size limit (collision.cu:121-159), split so that contacts can be spread over threads:
// step_limit_base is the per-segment start value, contact_step_limit one contact's bound
// 0.45 x centre-line distance.  A contact also stages the partner's endpoints relative to p0
// in slot `stage` of relA/relB (read by every Newton iteration of the substep; NO_STAGE: not
// staged), reports an interpenetration (distance at or below 2 radius, each unordered pair
// once, o > k) and returns the centre-line distance in dist.
constexpr size_t NO_STAGE = ~(size_t)0;

template <typename R>
__device__ __forceinline__ R step_limit_base(const Dev<R>& d, int k, const SceneParams<R>& sp) {
    typedef Ex<R> E;
    R m = sp.stepBase;
    if (sp.useVelRadius) m = E::add(m, E::sqrt(xlen2(xyz(d.dx[0][k].a))));
    return m;
}

template <typename R>
__device__ __forceinline__ R contact_step_limit(const Dev<R>& d, int k, size_t stage, int o, const V3<R>& a0,
                                                const V3<R>& a1, const SceneParams<R>& sp, bool& pen, R& dist) {
    typedef Ex<R> E;
    const V3<R> b0 = xsub(xyz(d.pos[o]), a0);
    const V3<R> b1 = xsub(xyz(d.pos[o + 1]), a0);
    if (stage != NO_STAGE) {
        d.relA[stage] = v4(b0, b1.x);
        R2<R> rb;
        rb.x = b1.y;
        rb.y = b1.z;
        d.relB[stage] = rb;
    }
    const UVT<R> uv = closest_uv_exact(a1, b0, b1);
    const V3<R> nrm = xsub(xscale(uv.u, a1), xmix(b0, b1, uv.v));
    const R l = E::sqrt(xlen2(nrm));
    if (stage != NO_STAGE && d.relD) {
        // The computed distance can lie above the true one by the rounding of the closest point's
        // parameter, 3 roundings of |b| over the sine of the angle: 5.7e-6 |b| in single precision (below a
        // sine of 0.03 the parameter is formed in FP64), 1e-8 |b| in double.  So does the Newton kernel's.
        const R b = (fabs(b0.x) + fabs(b0.y) + fabs(b0.z)) + (fabs(b1.x) + fabs(b1.y) + fabs(b1.z));
        const R room = l - (sp.outOfRange + R(sizeof(R) == 4 ? 2e-5 : 1e-7) * b);
        d.relD[stage] = room > R(0) ? room * room : R(-1);
    }
    pen = o > k && l <= sp.twoR;
    dist = l;
    const R safe = E::mul(E::sub(R(1), R(0.1f)), R(0.5f));
    return E::mul(safe, l);
}

// Minimum of step limits in shared memory: they are >= 0, so their bits order like them (and those of
// something that is not a number are larger than infinity's: it is passed over, as in ymin).
__device__ __forceinline__ void limit_min(float* at, float v) {
    atomicMin(reinterpret_cast<unsigned*>(at), __float_as_uint(v));
}
__device__ __forceinline__ void limit_min(double* at, double v) {
    atomicMin(reinterpret_cast<unsigned long long*>(at), (unsigned long long)__double_as_longlong(v));
}

}  // namespace yb
