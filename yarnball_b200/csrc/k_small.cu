// k_small.cu - one thread block advances a small simulation through every substep of an
// advance() in a single launch.
//
// A scene of a few hundred vertices keeps a B200 busy for microseconds per kernel, so the
// per-substep kernel sequence is bound by launch latency.  Here one block runs all substeps,
// with the whole state, the contact lists and the staged partner positions in shared memory:
// global memory is read at the start and written at the end.  The device functions are the
// multi-block kernels' (step.cuh, detect.cuh), given a copy of the engine's pointers that
// points into shared memory.
//
// The block is bound by the latency of its dependent chain, not by issue, so the chain is
// shortened and split over roles:
//   * `vt` vertex threads (one vertex each) and CT contact threads.  In a Newton iteration the
//     contact threads evaluate the contacts, CT at a time and one per thread, while the vertex
//     threads evaluate inertia, glue and stretch, then sum the contributions in list order, add the own
//     terms (after the contacts, so that large opposite contact forces cancel first: up to 1 % slower than
//     before them) and solve, beside the bending gradients of the contact threads; the next iteration's contacts
//     start as soon as the new displacements are known, beside the orientation update;
//   * the pair search tests all padded boxes, every pair of vertices once, spread over all
//     threads; hits go through a queue per warp so that the exact narrow phase runs on 32 pairs
//     at once;
//   * contact lists are rows of a bit matrix: a kept pair sets two bits, and reading a row
//     upwards gives the list in partner order without a sort.
// Measured (B200, us per substep, before -> now, where before one thread ran each vertex with
// all of its pairs and contacts in global memory): README scene (64 vertices, few contacts)
// 53 -> 15; swatch of 216 vertices (2 contacts a segment) 209 -> 46.  Testing contacts for being out of
// range first, as k_iter_bal does: 46 -> 45, but 15 -> 16 in the README scene.
//
// Reference semantics: Sim::advance (sim/step.cpp:36-55) with initItr / endItr
// (sim/iteration.cu), detectCollisions + buildCollisionList (sim/collision.cu:39-119),
// recomputeStepLimitKernel (collision.cu:121-159), cosseratItr + quaternionLambdaItr
// (sim/cosserat.cu).
#include "step.cuh"

namespace yb {

constexpr int SMALL_VERTS = 256;  // largest simulation this path runs (vertices)
constexpr int SMALL_WORDS = SMALL_VERTS / 32;
constexpr int SMALL_SCENES = 16;  // scene parameters kept in shared memory up to this many

template <typename R>
struct SmallShare {
    static constexpr int CT = sizeof(R) == 4 ? 256 : 128;   // contact threads
    static constexpr int CAP = sizeof(R) == 4 ? 2560 : 640; // contacts held here; the rest is read from global memory
    static constexpr int WARPS = (SMALL_VERTS + CT) / 32;
    V4<R> pos[SMALL_VERTS], posC[SMALL_VERTS], vel[SMALL_VERTS], lastVel[SMALL_VERTS];
    V4<R> q[2][SMALL_VERTS], qRest[SMALL_VERTS];
    D2<R> dx[2][SMALL_VERTS];
    VP<R> vp[SMALL_VERTS];
    R stepLim[SMALL_VERTS];
    V4<R> con4[2][4][CT];  // contributions of a chunk of contacts, as k_iter_bal groups them
    R2<R> con2[2][CT];
    V4<R> relA[CAP];
    R2<R> relB[CAP];
    int pack[CAP];         // owner << 16 | partner
    R halo[10][SMALL_VERTS];  // each vertex's own terms, then fb, Hb and the step limit of each segment
    V4<R> bend[SMALL_VERTS];  // gradient of each segment's bending terms
    float4 boxLo[SMALL_VERTS], boxHi[SMALL_VERTS];
    unsigned adj[SMALL_VERTS][SMALL_WORDS];
    int queue[WARPS][64];
    int warpSum[SMALL_WORDS];
    SceneParams<R> sp[SMALL_SCENES];
};

template <typename R>
__global__ void __launch_bounds__(SMALL_VERTS + SmallShare<R>::CT)
    k_small(const __grid_constant__ Dev<R> g, const SceneParams<R>* params, int* errOut, int steps, int numItr,
            unsigned long long step0, int detectionPeriod, int kahan) {
    constexpr int CT = SmallShare<R>::CT, CAP = SmallShare<R>::CAP;
    const unsigned FULL = 0xffffffffu;
    extern __shared__ __align__(16) unsigned char raw[];
    SmallShare<R>& m = *reinterpret_cast<SmallShare<R>*>(raw);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const int n = g.n;
    const int vt = (int)blockDim.x - CT;  // vertex threads: n rounded up to whole warps
    const int k = t;
    const bool vertexWarp = t < vt, valid = t < n;
    Dev<R> d = g;
    d.pos = m.pos; d.posC = m.posC; d.vel = m.vel; d.lastVel = m.lastVel;
    d.dx[0] = m.dx[0]; d.dx[1] = m.dx[1];
    d.q[0] = m.q[0]; d.q[1] = m.q[1];
    d.qRest = m.qRest; d.vp = m.vp; d.stepLim = m.stepLim;
    d.relA = m.relA; d.relB = m.relB; d.relD = nullptr; d.relCap = CAP;
    {
        // word by word, so that a whole warp reads host memory at once
        static_assert(sizeof(SceneParams<R>) % 8 == 0, "parameters are copied by 8 bytes");
        const int words = g.numScenes * (int)(sizeof(SceneParams<R>) / 8);
        const bool here = g.numScenes <= SMALL_SCENES;
        const unsigned long long* from = reinterpret_cast<const unsigned long long*>(params ? params : g.sp);
        unsigned long long* keep = reinterpret_cast<unsigned long long*>(const_cast<SceneParams<R>*>(g.sp));
        unsigned long long* to = reinterpret_cast<unsigned long long*>(m.sp);
        for (int i = t; i < words; i += blockDim.x) {
            const unsigned long long w = from[i];
            if (params) keep[i] = w;
            if (here) to[i] = w;
        }
        if (here) d.sp = m.sp;
    }
    uint32_t fl0 = 0;
    int nc = 0;
    if (valid) {
        m.pos[k] = g.pos[k]; m.posC[k] = g.posC[k]; m.vel[k] = g.vel[k]; m.lastVel[k] = g.lastVel[k];
        m.q[0][k] = g.q[0][k]; m.q[1][k] = g.q[0][k]; m.qRest[k] = g.qRest[k];
        m.dx[0][k] = g.dx[0][k]; m.dx[1][k] = g.dx[1][k];
        const VP<R> vp = g.vp[k];
        m.vp[k] = vp;
        fl0 = vp.flags;
        // the lists of the last detection, in case the first substep does not detect
        nc = min(max(g.numCols[k], 0), MAX_COLS);
    }
    if (vertexWarp) {
        m.stepLim[k] = yinf<R>();
#pragma unroll
        for (int w = 0; w < SMALL_WORDS; w++) m.adj[k][w] = 0u;
        for (int c = 0; c < nc; c++) {
            const int j = g.cols[col_at(k, c)];
            if ((unsigned)j < (unsigned)n) m.adj[k][j >> 5] |= 1u << (j & 31);
        }
    }
    const bool seg = valid && (fl0 & F_HAS_NEXT);
    const int sc = scene_of(fl0);
    __syncthreads();

    int off = 0, total = 0;  // this segment's first packed contact; all contacts
    int pens = 0, most = 0;
    float dmin = INFINITY;
    bool lists = false;      // the packed contacts follow the bit matrix
    for (int s = 0; s < steps; s++) {
        if (valid) init_vertex(d, k);
        __syncthreads();
        const bool detect = detectionPeriod > 0 && (step0 + (unsigned long long)s) % (unsigned long long)detectionPeriod == 0;
        if (detect) {
            if (vertexWarp) {
                float4 lo = empty_lo(), hi = empty_hi();
                if (seg) {
                    R reach;
                    float_box(segment_box(d, k, d.sp[sc], reach), lo, hi);
                    lo.w = __int_as_float(sc);
                }
                m.boxLo[k] = lo;
                m.boxHi[k] = hi;
#pragma unroll
                for (int w = 0; w < SMALL_WORDS; w++) m.adj[k][w] = 0u;
            }
            __syncthreads();
            // vertex x against x + o (cyclic), o = 1 .. n / 2: every pair of vertices once
            int qn = 0;
            int* queue = m.queue[warp];
            auto drain = [&](int first, int count) {
                if (lane < count) {
                    const int e = queue[first + lane];
                    const int x = e >> 16, y = e & 0xffff;
                    if (pair_keep(d, x, y, d.sp[scene_of(m.vp[x].flags)])) {
                        atomicOr(&m.adj[x][y >> 5], 1u << (y & 31));
                        atomicOr(&m.adj[y][x >> 5], 1u << (x & 31));
                    }
                }
                __syncwarp();
            };
            const int parts = (int)blockDim.x / vt, part = t / vt;
            if (part < parts) {  // whole warps
                const int x = t - part * vt;
                const float4 lo = x < n ? m.boxLo[x] : empty_lo(), hi = x < n ? m.boxHi[x] : empty_hi();
                const int half = n / 2;
                // 32 partners at a time into a mask, then one hit of each thread at a time
                for (int o0 = 1 + part; o0 <= half; o0 += 32 * parts) {
                    unsigned hits = 0;
                    const int count = min(32, (half - o0) / parts + 1);
#pragma unroll 4
                    for (int i = 0; i < count; i++) {
                        int y = x + o0 + i * parts;
                        if (y >= n) y -= n;
                        y = min(y, SMALL_VERTS - 1);  // threads past the last vertex read, and meet nothing
                        if (boxes_meet(lo, hi, m.boxLo[y], m.boxHi[y])) hits |= 1u << i;
                    }
                    // with n even, x and x + n / 2 meet from both sides
                    if (2 * (o0 + (count - 1) * parts) == n && x >= half) hits &= ~(1u << (count - 1));
                    while (__any_sync(FULL, hits != 0)) {
                        int y = x + o0 + (__ffs(hits) - 1) * parts;
                        if (y >= n) y -= n;
                        const int a = min(x, y), b = max(x, y);
                        const bool take = hits && b - a > 2 && __float_as_int(lo.w) == __float_as_int(m.boxLo[y].w);
                        hits &= hits - 1;
                        const unsigned mask = __ballot_sync(FULL, take);
                        if (take) queue[qn + __popc(mask & lt)] = a << 16 | b;
                        qn += __popc(mask);
                        __syncwarp();
                        if (qn >= 32) {
                            qn -= 32;
                            drain(qn, 32);
                        }
                    }
                }
                if (qn) drain(0, qn);
            }
            __syncthreads();
            lists = false;
        }
        if (!lists) {
            // list lengths, their clamp (the lowest partner ids stay) and the packed contacts
            if (vertexWarp) {
                int c = 0;
#pragma unroll
                for (int w = 0; w < SMALL_WORDS; w++) c += __popc(m.adj[k][w]);
                if (detect) {
                    most = max(most, c);
                    if (c > MAX_COLS) g.err[EW_ERROR] = 1;
                }
                nc = min(c, MAX_COLS);
                off = nc;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(FULL, off, o);
                    if (lane >= o) off += y;
                }
                if (lane == 31) m.warpSum[warp] = off;
                off -= nc;
            }
            __syncthreads();
            total = 0;
            for (int w = 0; w < vt / 32; w++) {
                if (w < warp && vertexWarp) off += m.warpSum[w];
                total += m.warpSum[w];
            }
            if (vertexWarp && nc) {
                int at = off;
                const int end = off + nc;
                for (int w = 0; w < SMALL_WORDS; w++)
                    for (unsigned bits = m.adj[k][w]; bits && at < end; bits &= bits - 1, at++) {
                        const int e = k << 16 | (32 * w + __ffs(bits) - 1);
                        if (at < CAP) m.pack[at] = e; else g.csrCols[at] = e;
                    }
            }
            lists = true;
        }
        if (seg) m.stepLim[k] = step_limit_base(d, k, d.sp[sc]);
        __syncthreads();
        // step limit, staged partner positions, interpenetration statistics
        for (int f = t; f < total; f += blockDim.x) {
            const int e = f < CAP ? m.pack[f] : g.csrCols[f];
            const int a = e >> 16, o = e & 0xffff;
            const V3<R> a0 = xyz(m.pos[a]);
            const V3<R> a1 = xsub(xyz(m.pos[a + 1]), a0);
            bool pen;
            R dist;
            const R lim = contact_step_limit(d, a, f < CAP ? (size_t)f : NO_STAGE, o, a0, a1,
                                             d.sp[scene_of(m.vp[a].flags)], pen, dist);
            pens += pen;
            dmin = fminf(dmin, (float)dist);
            limit_min(&m.stepLim[a], lim);
        }
        __syncthreads();
        if (valid && !(seg && d.sp[sc].useStepLimit)) m.stepLim[k] = yinf<R>();

        const int chunks = (total + CT - 1) / CT;
        const bool bendHere = chunks == 0;  // else the contact threads have no time to spare
        int buf = 0;
        OwnTerms<R> own;
        own.flags = 0;
        own.invMass = R(0);
        own.sl = yinf<R>();
        V3<R> p0(R(0)), e(R(0));
        if (valid) {
            own = own_terms(d, k, d.sp[sc]);
            p0 = xyz(m.pos[k]);
            if (seg) e = xyz(m.pos[k + 1]) - p0;
        }
        for (int it = 0; it < numItr; it++) {
            const int src = it & 1;
            const D2<R>* DX = m.dx[src];
            const V4<R>* QO = m.q[src];
            auto evaluate = [&](int chunk, int to) {
                const int u = t - vt, f = chunk * CT + u;
                if (u < 0 || f >= total) return;
                const int e = f < CAP ? m.pack[f] : g.csrCols[f];
                const int a = e >> 16, o = e & 0xffff;
                const V3<R> a0 = xyz(m.pos[a]);
                V3<R> r0, r1;
                partner_rel(d, (unsigned)f, o, a0, r0, r1);
                const D2<R> ad = DX[a], pd = DX[o];
                V3<R> fa(R(0)), fb(R(0));
                H3<R> Ha, Hb;
                Ha.zero();
                Hb.zero();
                contact_term(xyz(m.pos[a + 1]) - a0, xyz(ad.a), xyz(ad.b), r0, r1, xyz(pd.a), xyz(pd.b),
                             d.sp[scene_of(m.vp[a].flags)], fa, Ha, fb, Hb);
                V4<R> w;
                w.x = fa.x; w.y = fa.y; w.z = fa.z; w.w = fb.x; m.con4[to][0][u] = w;
                w.x = fb.y; w.y = fb.z; w.z = Ha.d[0]; w.w = Ha.d[1]; m.con4[to][1][u] = w;
                w.x = Ha.d[2]; w.y = Ha.d[3]; w.z = Ha.d[4]; w.w = Ha.d[5]; m.con4[to][2][u] = w;
                w.x = Hb.d[0]; w.y = Hb.d[1]; w.z = Hb.d[2]; w.w = Hb.d[3]; m.con4[to][3][u] = w;
                R2<R> w2;
                w2.x = Hb.d[4]; w2.y = Hb.d[5];
                m.con2[to][u] = w2;
            };
            V3<R> fa(R(0)), fb(R(0));
            H3<R> Ha, Hb;
            Ha.zero();
            Hb.zero();
            R sl = own.sl;
            Q<R> q0 = qmk(R(0), R(0), R(0), R(1));
            V3<R> dx(R(0));
            if (chunks) evaluate(0, buf);
            // The own terms wait for the contacts in rows of the halo, which are free until then: in registers
            // they make the FP64 build spill (216 vertices: 92 us a substep, 84 this way).
            if (vertexWarp) {
                OwnSums<R> mine{V3<R>(R(0)), V3<R>(R(0)), R(0), R(0)};
                if (valid) {
                    const D2<R> ad = DX[k];
                    dx = xyz(ad.a);
                    q0 = qof(QO[k]);
                    mine = own_sums(d, own, DX, d.sp[sc].D, p0, e, dx, xyz(ad.b), q0);
                }
                m.halo[0][k] = mine.fa.x; m.halo[1][k] = mine.fa.y; m.halo[2][k] = mine.fa.z;
                m.halo[3][k] = mine.fb.x; m.halo[4][k] = mine.fb.y; m.halo[5][k] = mine.fb.z;
                m.halo[6][k] = mine.ha; m.halo[7][k] = mine.hb;
            }
            for (int c = 0; c < max(chunks, 1); c++, buf ^= 1) {
                // chunk c is evaluated, chunk c - 1 summed, and the rotors are those of the last iteration
                __syncthreads();
                if (c + 1 < chunks)
                    evaluate(c + 1, buf ^ 1);
                else if (bendHere)
                    for (int i = t - vt; i < n; i += CT)
                        if (i >= 0) {
                            const uint32_t fl = m.vp[i].flags;
                            if (turns(fl)) m.bend[i] = v4of(bending_gradient(d, i, QO, fl, qof(QO[i])));
                        }
                if (vertexWarp && c < chunks) {
                    const int f1 = min(off + nc, (c + 1) * CT) - c * CT;
                    for (int i = max(off - c * CT, 0); i < f1; i++) {
                        const V4<R> w0 = m.con4[buf][0][i], w1 = m.con4[buf][1][i], w2 = m.con4[buf][2][i],
                                    w3 = m.con4[buf][3][i];
                        const R2<R> w4 = m.con2[buf][i];
                        fa += V3<R>(w0.x, w0.y, w0.z);
                        fb += V3<R>(w0.w, w1.x, w1.y);
                        Ha.d[0] += w1.z; Ha.d[1] += w1.w;
                        Ha.d[2] += w2.x; Ha.d[3] += w2.y; Ha.d[4] += w2.z; Ha.d[5] += w2.w;
                        Hb.d[0] += w3.x; Hb.d[1] += w3.y; Hb.d[2] += w3.z; Hb.d[3] += w3.w;
                        Hb.d[4] += w4.x; Hb.d[5] += w4.y;
                    }
                }
            }
            V3<R> dxn = dx;
            if (vertexWarp) {
                // own terms after the contacts, as in the multi-block kernels: large opposite contact forces
                // cancel first
                fa += V3<R>(m.halo[0][k], m.halo[1][k], m.halo[2][k]);
                fb += V3<R>(m.halo[3][k], m.halo[4][k], m.halo[5][k]);
                Ha.add_diag(m.halo[6][k]);
                Hb.add_diag(m.halo[7][k]);
                m.halo[0][k] = fb.x; m.halo[1][k] = fb.y; m.halo[2][k] = fb.z;
#pragma unroll
                for (int q = 0; q < 6; q++) m.halo[3 + q][k] = Hb.d[q];
                m.halo[9][k] = sl;
                asm volatile("bar.sync 1, %0;" ::"r"(vt) : "memory");  // the vertex threads only
                if (valid) {
                    if (own.flags & F_HAS_PREV) {
                        fa += V3<R>(m.halo[0][k - 1], m.halo[1][k - 1], m.halo[2][k - 1]);
                        H3<R> hp;
#pragma unroll
                        for (int q = 0; q < 6; q++) hp.d[q] = m.halo[3 + q][k - 1];
                        Ha.add(hp);
                        sl = ymin(sl, m.halo[9][k - 1]);
                    }
                    if (own.invMass != R(0)) {
                        dxn = dx + d.sp[sc].accel * solve3(Ha, fa);
                        const R l = len(dxn);
                        if (l > sl && l > R(0)) dxn *= sl / l;
                    }
                    // the new iterate pair: this vertex's half of its own and of the one before
                    m.dx[src ^ 1][k].a = v4(dxn, R(0));
                    if (k > 0) m.dx[src ^ 1][k - 1].b = v4(dxn, R(0));
                    if (k == n - 1) m.dx[src ^ 1][k].b = v4(V3<R>(R(0)), R(0));
                }
            }
            __syncthreads();
            if (valid) {
                if (turns(own.flags))
                    q0 = turned(q0, bendHere ? qof(m.bend[k]) : bending_gradient(d, k, QO, own.flags, q0), e, dxn, xyz(m.dx[src ^ 1][k].b), own.invl, own.kStretch);
                m.q[src ^ 1][k] = v4of(q0);
            }
        }
        if (numItr & 1) {
            __syncthreads();  // neighbours still read q[0], which end_vertex overwrites
            if (valid) end_vertex(d, k, 1, 1, kahan);
        } else if (valid) {
            end_vertex(d, k, 0, 0, kahan);
        }
        __syncthreads();
    }

    if (valid) {
        g.pos[k] = m.pos[k]; g.posC[k] = m.posC[k]; g.vel[k] = m.vel[k]; g.lastVel[k] = m.lastVel[k];
        g.q[0][k] = m.q[0][k]; g.dx[0][k] = m.dx[0][k]; g.dx[1][k] = m.dx[1][k];
        g.stepLim[k] = m.stepLim[k];
        g.numCols[k] = nc;
        int c = 0;
        for (int w = 0; w < SMALL_WORDS; w++)
            for (unsigned bits = m.adj[k][w]; bits && c < nc; bits &= bits - 1)
                g.cols[col_at(k, c++)] = 32 * w + __ffs(bits) - 1;
    }
    if (most) atomicMax(&g.err[EW_MAX_COLS], most);
    if (pens) {
        atomicAdd(&g.err[EW_PENETRATIONS], pens);
        g.err[EW_WARNING] = 2;
    }
    if (dmin < INFINITY) atomicMin(&g.err[EW_MIN_DIST], __float_as_int(dmin));
    __syncthreads();
    if (t < EW_COUNT) errOut[t] = __ldcg(g.err + t);
}

template <typename R>
bool small_path_fits(const Dev<R>& d) {
    return d.n > 0 && d.n <= SMALL_VERTS;
}

template <typename R>
cudaError_t small_path_prepare() {
    static_assert(sizeof(SmallShare<R>) <= 227 * 1024, "shared memory of one block");
    return cudaFuncSetAttribute(k_small<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmallShare<R>));
}

template <typename R>
void launch_small(const Dev<R>& d, const SceneParams<R>* params, int* errOut, int steps, int numItr,
                  unsigned long long step0, int detectionPeriod, bool kahan, cudaStream_t s) {
    if (d.n <= 0 || steps <= 0) return;
    const int threads = (d.n + 31) / 32 * 32 + SmallShare<R>::CT;
    k_small<R><<<1, threads, sizeof(SmallShare<R>), s>>>(d, params, errOut, steps, numItr, step0, detectionPeriod, kahan ? 1 : 0);
}

#define YB_INST(R)                                                                                            \
    template bool small_path_fits<R>(const Dev<R>&);                                                          \
    template cudaError_t small_path_prepare<R>();                                                             \
    template void launch_small<R>(const Dev<R>&, const SceneParams<R>*, int*, int, int, unsigned long long, int, bool, \
                                  cudaStream_t);
YB_INST(float)
YB_INST(double)

}  // namespace yb
