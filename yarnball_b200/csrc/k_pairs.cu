// k_pairs.cu - broadphase over clusters of 32 curve-consecutive segments.
//
// The reference calls an LBVH library (call sites KittenEngine/YarnBall/sim/collision.cu:94-119);
// what it keeps of the result is the set of pairs that pass the narrow-phase filter
// (detect.cuh), so any enumeration that visits every pair of overlapping padded boxes gives
// the same contact lists.  Here:
//   * at a rebuild the segments of every scene are sorted along a Hilbert curve (k_bvh.cu);
//     32 consecutive ones are a cluster.  Consecutive cells of that curve are neighbours, so a
//     run of 32 has a compact box (a run along the Morton curve can jump across the scene);
//   * k_boxes, every detection: the padded box of every segment in curve order, its cluster's
//     box, and the boxes of 32, 1024 and 32768 clusters (levels 1-3, as many as the scene needs
//     to end with at most 32 nodes);
//   * k_pairs: a warp takes one cluster, tests its box against 32 nodes of a level at a time
//     (one per lane, two coalesced loads), descends where they overlap, and for each
//     overlapping cluster tests segments against segments.
// Positions in the tree follow from the counts alone: a node's children are the 32 nodes below
// it, so there are no links, no per-node arrival counters in the leaves' path and no chain of
// dependent loads per segment; a walk is paid once per 32 segments.
//
// Measured (B200, per detection, refit + walk of the BVH before -> boxes + pairs): 8.4M vertices
// in 269 scenes, 3.2 contacts a segment: 1.27 + 3.9 ms -> 0.17 + 2.2 ms; one pile of 65,792
// vertices, 11.5 contacts: 49 + 280 us -> 10 + 75 us; a swatch of 1,949 vertices: 32 + 78 us -> 7 + 12 us.
//
// Boxes are kept in single precision in both builds: in the FP64 one segments' boxes are rounded
// outwards, and those of nodes to nearest (bounds() reports their union) and widened by a float where
// they are tested.  A tested box may only be too large, and what it lets through the filter decides.
#include "detect.cuh"

namespace yb {

// Order-preserving map of floats to unsigned, so that a warp's minimum is one redux.
__device__ __forceinline__ unsigned box_ord(float f) {
    const unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float box_unord(unsigned u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}
__device__ __forceinline__ float warp_min(float f) {
    return box_unord(__reduce_min_sync(0xffffffffu, box_ord(f)));
}
__device__ __forceinline__ float warp_max(float f) {
    return box_unord(__reduce_max_sync(0xffffffffu, box_ord(f)));
}
__device__ __forceinline__ void warp_box(float4& lo, float4& hi) {
    lo.x = warp_min(lo.x); lo.y = warp_min(lo.y); lo.z = warp_min(lo.z);
    hi.x = warp_max(hi.x); hi.y = warp_max(hi.y); hi.z = warp_max(hi.z);
}
// One block per level-1 node (32 clusters, one per warp).  The block writes its clusters' boxes
// and their union; the block that completes a level-2 (level-3) node, told by an arrival
// counter that wraps to zero, writes that node's box from its 32 children.  Bound by the
// gathers of positions and predicted displacements (64 bytes a segment in curve order) and the
// 32 bytes written.
constexpr int BOX_THREADS = 1024;

template <typename R>
__global__ void __launch_bounds__(BOX_THREADS) k_boxes(Dev<R> d, const int* __restrict__ sortedVals) {
    after_previous_kernel();
    __shared__ float4 sLo[32], sHi[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int s = d.l1Scene[blockIdx.x];
    const SceneClus sc = d.sceneClus[s];
    const int n1 = (int)blockIdx.x - sc.lvl[1];  // level-1 node within the scene
    const int c = 32 * n1 + w;                   // cluster within the scene
    float4 lo = empty_lo(), hi = empty_hi();
    if (c < sc.count[0]) {
        const int p = 32 * c + lane;
        const size_t at = 32 * (size_t)(sc.lvl[0] + c) + lane;
        if (p < sc.segCount) {
            const int k = sortedVals[sc.segBase + p];
            R reach;
            const Box<R> b = segment_box(d, k, d.sp[s], reach);
            float4 slo, shi;
            float_box(b, slo, shi);
            slo.w = __int_as_float(k);
            shi.w = (float)reach;
            d.leafLo[at] = slo;
            d.leafHi[at] = shi;
            nearest_box(b, lo, hi);
        } else {
            d.leafLo[at] = empty_lo();
            d.leafHi[at] = empty_hi();
        }
        warp_box(lo, hi);
        if (lane == 0) {
            d.lvlLo[0][sc.lvl[0] + c] = lo;
            d.lvlHi[0][sc.lvl[0] + c] = hi;
        }
    }
    if (lane == 0) {
        sLo[w] = lo;
        sHi[w] = hi;
    }
    __syncthreads();
    if (w != 0) return;
    lo = sLo[lane];
    hi = sHi[lane];
    warp_box(lo, hi);
    int node = n1;
    for (int level = 1;; level++) {
        if (lane == 0) {
            d.lvlLo[level][sc.lvl[level] + node] = lo;
            d.lvlHi[level][sc.lvl[level] + node] = hi;
        }
        if (level >= sc.top) return;
        const int parent = node >> 5;
        const int kids = min(32, sc.count[level] - 32 * parent);
        unsigned last = 0;
        if (lane == 0) {
            __threadfence();  // this node's box before the arrival
            last = atomicInc(d.lvlCount[level + 1] + sc.lvl[level + 1] + parent, (unsigned)(kids - 1)) ==
                   (unsigned)(kids - 1);
            __threadfence();  // the siblings' boxes after it
        }
        if (!__shfl_sync(0xffffffffu, last, 0)) return;
        lo = empty_lo();
        hi = empty_hi();
        if (lane < kids) {
            lo = __ldcg(d.lvlLo[level] + sc.lvl[level] + 32 * parent + lane);
            hi = __ldcg(d.lvlHi[level] + sc.lvl[level] + 32 * parent + lane);
        }
        warp_box(lo, hi);
        node = parent;
    }
}

// Pair search.  Each cluster is searched by `parts` warps; all of them walk the levels, and
// cluster j >= i of a walk is worked by warp (j - i) mod parts, so that a scene of a few
// thousand segments still spreads over the chip.  For a pair of clusters, the segments of each
// that reach the other's box are found by ballots; the fewer of the two sides are packed in
// shared memory and every lane tests its own segment against them in a loop (two broadcast
// 16-byte reads and six compares a test), collecting the hits in a bit mask.  Hits go through a
// queue of the warp, so that the separately rounded narrow-phase test runs on 32 pairs at once.
// Bound by issue and latency.  `parts` makes 96 warps for every SM, three times what an SM holds, since the
// clusters' work is uneven (blocks of 4 warps: this kernel and the list pass take 330 / 232 / 222 us
// with 32 / 96 / 192 warps per SM on a bundle of 100,352 vertices, 144 / 146 / 163 us on a pile
// of 65,792 and 365 / 342 / 361 us on one of 262,144; every part repeats the walk).
constexpr int PAIR_THREADS = 32;  // a warp to a block: the clusters' work is uneven, and a block holds its
                                  // place on the SM until its last warp is done (128 threads: 20 % longer)

struct PairShare {
    float4 lo[32], hi[32];
    int qx[64], qy[64];      // queued pairs
    float qrx[64], qry[64];  // ... and the segments' reaches (used by the FP32 build)
};

// Narrow phase of m queued pairs, one per lane; kept ones go to both lists.  Not inlined: its
// registers would otherwise be held back from every warp of the search.
template <typename R>
__device__ __noinline__ void pairs_filter(const Dev<R>& d, const PairShare& sh, int first, int m, int s) {
    const int lane = threadIdx.x;
    if (lane < m) {
        const int a = sh.qx[first + lane], b = sh.qy[first + lane];
        const int x = min(a, b), y = max(a, b);
        const SceneParams<R>& sp = d.sp[s];
        R rx, ry;  // added in the order x, y: the filter distance is rounded as pair_keep's
        if constexpr (sizeof(R) == 4) {
            const float ra = sh.qrx[first + lane], rb = sh.qry[first + lane];
            rx = a < b ? ra : rb;
            ry = a < b ? rb : ra;
        } else {
            rx = sp.useVelRadius ? segment_reach(d, x) : R(0);
            ry = sp.useVelRadius ? segment_reach(d, y) : R(0);
        }
        if (pair_within(pair_distance2(d, x, y), rx, ry, sp) && !(d.sceneGlued[s] && pair_joined(d, x, y))) {
            list_append(d, x, y);
            list_append(d, y, x);
        }
    }
    __syncwarp();
}

template <typename R>
__global__ void __launch_bounds__(PAIR_THREADS, 32) k_pairs(const __grid_constant__ Dev<R> d, int parts) {
    after_previous_kernel();
    const unsigned FULL = 0xffffffffu;
    __shared__ PairShare sh;
    const int lane = threadIdx.x;
    const unsigned lt = (1u << lane) - 1u;
    const int gw = (int)blockIdx.x;
    const int ci = gw / parts, part = gw - ci * parts;
    if (ci >= d.nclus) return;
    const int s = d.clusScene[ci];
    const SceneClus& sc = d.sceneClus[s];
    const int base0 = sc.lvl[0], top = sc.top;
    const int i = ci - base0;
    const float4 alo = d.leafLo[32 * (size_t)ci + lane], ahi = d.leafHi[32 * (size_t)ci + lane];
    float4 ulo = d.lvlLo[0][ci], uhi = d.lvlHi[0][ci];
    widen_box<R>(ulo, uhi);
    int qn = 0;  // queued pairs (identical in every lane)

    // lanes (own box, own segment) against the r boxes packed in sh.lo / sh.hi
    auto packed_hits = [&](const float4& olo, const float4& ohi, int r) {
        unsigned hits = 0;
#pragma unroll 4
        for (int t = 0; t < r; t++)
            if (boxes_meet(sh.lo[t], sh.hi[t], olo, ohi)) hits |= 1u << t;
        return hits;
    };
    // clusters i and j >= i
    auto cross = [&](int j, const float4& blo, const float4& bhi) {
        float4 vlo = d.lvlLo[0][base0 + j], vhi = d.lvlHi[0][base0 + j];
        widen_box<R>(vlo, vhi);
        // the places past a scene's last segment hold none, whatever the boxes say
        const bool ha = __float_as_int(alo.w) >= 0 && boxes_meet(alo, ahi, vlo, vhi);
        const bool hb = __float_as_int(blo.w) >= 0 && boxes_meet(blo, bhi, ulo, uhi);
        const unsigned ma = __ballot_sync(FULL, ha), mb = __ballot_sync(FULL, hb);
        if (!ma || !mb) return;
        unsigned hits;
        float own, ownReach;
        if (__popc(ma) <= __popc(mb)) {
            if (ha) {
                const int r = __popc(ma & lt);
                sh.lo[r] = alo;
                sh.hi[r] = ahi;
            }
            __syncwarp();
            hits = packed_hits(blo, bhi, __popc(ma));
            if (!hb) hits = 0;
            // a pair inside the cluster is taken once: from the later of the two lanes
            if (j == i) hits &= (1u << __popc(ma & lt)) - 1u;
            own = blo.w;
            ownReach = bhi.w;
        } else {
            if (hb) {
                const int r = __popc(mb & lt);
                sh.lo[r] = blo;
                sh.hi[r] = bhi;
            }
            __syncwarp();
            hits = packed_hits(alo, ahi, __popc(mb));
            if (!ha) hits = 0;
            own = alo.w;
            ownReach = ahi.w;
        }
        // one hit of each lane at a time into the queue; neighbours on a yarn, whose boxes always
        // meet, are no contacts
        while (__any_sync(FULL, hits != 0)) {
            const int t = hits ? __ffs(hits) - 1 : 0;
            const int a = __float_as_int(own), b = __float_as_int(sh.lo[t].w);
            const bool take = hits && abs(a - b) > 2;
            hits &= hits - 1;
            const unsigned m = __ballot_sync(FULL, take);
            if (take) {
                const int at = qn + __popc(m & lt);
                sh.qx[at] = a;
                sh.qy[at] = b;
                if constexpr (sizeof(R) == 4) {
                    sh.qrx[at] = ownReach;
                    sh.qry[at] = sh.hi[t].w;
                }
            }
            qn += __popc(m);
            __syncwarp();
            if (qn >= 32) {
                qn -= 32;
                pairs_filter(d, sh, qn, 32, s);
            }
        }
        __syncwarp();
    };
    // overlap of this cluster's box with nodes base .. base + 31 of a level, those at or after it
    auto meet = [&](int level, int base) {
        const int at = base + lane;
        bool hit = false;
        if (at < sc.count[level] && at >= (i >> (5 * level))) {
            float4 lo = d.lvlLo[level][sc.lvl[level] + at], hi = d.lvlHi[level][sc.lvl[level] + at];
            widen_box<R>(lo, hi);
            hit = boxes_meet(lo, hi, ulo, uhi);
        }
        return __ballot_sync(FULL, hit);
    };

    unsigned m3 = top >= 3 ? meet(3, 0) : 1u;
    while (m3) {
        const int n3 = __ffs(m3) - 1;
        m3 &= m3 - 1;
        unsigned m2 = top >= 2 ? meet(2, 32 * n3) : 1u;
        while (m2) {
            const int n2 = 32 * n3 + __ffs(m2) - 1;
            m2 &= m2 - 1;
            unsigned m1 = top >= 1 ? meet(1, 32 * n2) : 1u;
            while (m1) {
                const int base = 32 * (32 * n2 + __ffs(m1) - 1);
                m1 &= m1 - 1;
                unsigned m0 = meet(0, base);
                if (parts > 1) m0 &= __ballot_sync(FULL, (unsigned)(base + lane - i) % (unsigned)parts == (unsigned)part);
                if (!m0) continue;
                // the next cluster's boxes are loaded while the current one is tested
                int j = base + __ffs(m0) - 1;
                const float4 *lo = d.leafLo + 32 * (size_t)base0 + lane, *hi = d.leafHi + 32 * (size_t)base0 + lane;
                float4 blo = lo[32 * (size_t)j], bhi = hi[32 * (size_t)j];
                while (m0) {
                    m0 &= m0 - 1;
                    const int jn = m0 ? base + __ffs(m0) - 1 : j;
                    float4 xlo = blo, xhi = bhi;
                    if (m0) {
                        xlo = lo[32 * (size_t)jn];
                        xhi = hi[32 * (size_t)jn];
                    }
                    cross(j, blo, bhi);
                    j = jn;
                    blo = xlo;
                    bhi = xhi;
                }
            }
        }
    }
    if (qn) pairs_filter(d, sh, 0, qn, s);
}

// Box of each scene: the union of its clusters' top level (at most 32 nodes; k_boxes must have run).
template <typename R>
__global__ void __launch_bounds__(32) k_scene_box(Dev<R> d, float* out) {
    const SceneClus sc = d.sceneClus[blockIdx.x];
    const int lane = threadIdx.x;
    float4 lo = empty_lo(), hi = empty_hi();
    if (lane < sc.count[sc.top]) {
        lo = d.lvlLo[sc.top][sc.lvl[sc.top] + lane];
        hi = d.lvlHi[sc.top][sc.lvl[sc.top] + lane];
    }
    warp_box(lo, hi);
    if (lane == 0) {
        float* o = out + 6 * (size_t)blockIdx.x;
        o[0] = lo.x; o[1] = lo.y; o[2] = lo.z;
        o[3] = hi.x; o[4] = hi.y; o[5] = hi.z;
    }
}

template <typename R>
void launch_boxes(const Dev<R>& d, cudaStream_t s) {
    if (d.nl1 > 0) launch_dependent(k_boxes<R>, d.nl1, BOX_THREADS, s, d, d.vals[0]);
}

template <typename R>
void launch_pairs(const Dev<R>& d, cudaStream_t s) {
    if (d.nclus <= 0) return;
    const int parts = min(32, (96 * d.sms + d.nclus - 1) / d.nclus);
    launch_dependent(k_pairs<R>, (size_t)d.nclus * parts, PAIR_THREADS, s, d, parts);
}

template <typename R>
void launch_cluster_box(const Dev<R>& d, float* out, cudaStream_t s) {
    k_scene_box<R><<<d.numScenes, 32, 0, s>>>(d, out);
}

#define YB_INST(R)                                               \
    template void launch_boxes<R>(const Dev<R>&, cudaStream_t);  \
    template void launch_pairs<R>(const Dev<R>&, cudaStream_t);  \
    template void launch_cluster_box<R>(const Dev<R>&, float*, cudaStream_t);
YB_INST(float)
YB_INST(double)

}  // namespace yb
