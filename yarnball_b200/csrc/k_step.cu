// k_step.cu - predictor, fused block-Jacobi Newton + orientation iteration, advection.
//
// Reference semantics (file:line in the reference project):
//   initItr               KittenEngine/YarnBall/sim/iteration.cu:7-41
//   cosseratItr           KittenEngine/YarnBall/sim/cosserat.cu:20-207
//   quaternionLambdaItr   KittenEngine/YarnBall/sim/cosserat.cu:209-253
//   endItr                KittenEngine/YarnBall/sim/iteration.cu:48-61
//
// Deliberate differences from the reference, all in the direction of determinism:
//   * strict Jacobi: iteration k reads only iteration k-1's dx and q (double buffers); the
//     reference updates both in place while neighbouring threads read them.
//   * one kernel per iteration does the position solve and the orientation update: a block
//     owns B-2 vertices and recomputes one halo segment on each side, so the orientation of
//     segment i sees the new dx of vertices i and i+1 without a second launch.
//   * contact lists are sorted by partner id, so force sums have a fixed order.
#include "step.cuh"

namespace yb {

template <typename R>
__global__ void __launch_bounds__(256) k_init(Dev<R> d, int clearLists) {
    after_previous_kernel();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.n) return;
    if (clearLists) d.numCols[i] = 0;
    init_vertex(d, i);
}

// ---------------------------------------------------------------------------------------
// Advection (iteration.cu:48-61) with Kahan-compensated position accumulation (FP32 build);
// also stores the start-of-substep velocity as lastVel (iteration.cu:19-20).
template <typename R>
__global__ void __launch_bounds__(256) k_end(Dev<R> d, int fb, int copyQ, int kahan) {
    after_previous_kernel();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.n) return;
    if (i <= list_tiles(d.n)) d.listStatus[i] = 0ull;  // for the next list pass (n is 3 or more)
    end_vertex(d, i, fb, copyQ, kahan);
}

// ---------------------------------------------------------------------------------------
// One block-Jacobi iteration: position solve (cosseratItr) then orientation update
// (quaternionLambdaItr), strict Jacobi.  A block has B vertex slots of T lanes each
// (NT = B*T threads): slot t handles vertex/segment k = b*(B-2)-1+t, writes it when
// t in [1, B-2] and only recomputes the halo slots t=0 and t=B-1.  The T lanes of a slot
// split the segment's contact loop (contacts s, s+T, ...) and combine their partial sums
// with an xor-shuffle butterfly, so every lane of the slot holds the identical total; the
// vertex solve and the orientation update are then evaluated by all T lanes and stored by
// lane 0.
template <typename R, int T>
__device__ __forceinline__ R slot_sum(R v) {
#pragma unroll
    for (int o = 1; o < T; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

template <typename R, int NT, int T, int MINB, bool PIPE>
__global__ void __launch_bounds__(NT, MINB) k_iter(Dev<R> d, int src) {
    constexpr int B = NT / T;
    constexpr int CORE = B - 2;
    const int t = threadIdx.x / T;
    const int lane = threadIdx.x % T;
    const int k = blockIdx.x * CORE - 1 + t;
    const int n = d.n;
    const bool valid = (k >= 0) && (k < n);
    const D2<R>* __restrict__ DX = d.dx[src];
    const V4<R>* __restrict__ QO = d.q[src];

    __shared__ R sFb[3][B];
    __shared__ R sHb[6][B];
    __shared__ R sSL[B];
    __shared__ R sDX[3][B];

    V3<R> fa(R(0)), fb(R(0));
    H3<R> Ha, Hb;
    Ha.zero(); Hb.zero();
    R sl = yinf<R>();
    uint32_t flags = 0;
    R invMass = R(0), lRest = R(1), kStretch = R(0);
    V3<R> p0(R(0)), p1(R(0)), dx(R(0)), dx1(R(0));
    Q<R> q0 = qmk(R(0), R(0), R(0), R(1));
    const SceneParams<R>* spp = d.sp;

    if (valid) {
        const VP<R> vp = d.vp[k];
        flags = vp.flags;
        lRest = vp.lRest;
        kStretch = vp.kStretch;
        spp = &d.sp[scene_of(flags)];
        const SceneParams<R>& sp = *spp;
        const V4<R> P = d.pos[k];
        p0 = xyz(P);
        invMass = P.w;
        const D2<R> own = DX[k];
        dx = xyz(own.a);
        dx1 = xyz(own.b);
        q0 = qof(QO[k]);
        const R D = sp.D;
        if (lane == 0) {
            if (invMass != R(0)) {
                // Inertia: H = m/h^2, f = m/h^2 (y - dx), y = h v + h^2 g (iteration.cu:26, cosserat.cu:40-45)
                const V4<R> v = d.vel[k];
                const R hh = sp.hh;
                const V3<R> y(sp.h * v.x + hh * sp.gx, sp.h * v.y + hh * sp.gy, sp.h * v.z + hh * sp.gz);
                Ha.diag(R(1) / (invMass * hh));
                fa = (R(1) / (hh * invMass)) * (y - dx);
            }
            if (vp.cid >= 0) {
                // Glue spring to the connected vertex (cosserat.cu:46-53)
                const R stiff = R(40);
                const V3<R> pc = xyz(d.pos[vp.cid]);
                const V3<R> dc = xyz(DX[vp.cid].a);
                fa -= stiff * ((p0 - pc) + (dx - dc) + D * dx);
                Ha.add_diag(stiff * (R(1) + D));
            }
        }
        if (flags & F_HAS_NEXT) {
            p1 = xyz(d.pos[k + 1]);
            sl = d.stepLim[k];
            if (lane == 0) {
                // Stretch-shear coupling to the segment orientation (cosserat.cu:63-81)
                const R invl = R(1) / lRest;
                const V3<R> c = ((p1 - p0) + (dx1 - dx)) * invl - qrotate(q0, V3<R>(R(1), R(0), R(0)));
                const R ks = kStretch * invl;
                R dd = ks * invl;
                fa += ks * c - (D * dd) * dx;
                fb += -ks * c - (D * dd) * dx1;
                dd *= R(1) + D;
                Ha.add_diag(dd);
                Hb.add_diag(dd);
            }
            // Barrier + friction over this lane's share of the contact list (packed slots).
            // Partner positions relative to p0 are staged per substep in the slots below
            // relCap; the partner's iterate pair is one 32-byte gather.
            // With PIPE the loads of the lane's next contact are issued before the current
            // contact's arithmetic, so the dependent partner gather overlaps it (more
            // registers); without it each contact loads then computes.
            unsigned off;
            const int nc = contact_range(d, k, off);
            const unsigned* __restrict__ cl = d.csrCols + off;
            const V3<R> e = p1 - p0;
            if constexpr (!PIPE) {
                for (int c2 = lane; c2 < nc; c2 += T) {
                    const int j = packed_partner(__ldg(cl + c2));
                    if (!partner_ok(d, j)) continue;
                    V3<R> r0, r1;
                    partner_rel(d, off + c2, j, p0, r0, r1);
                    const D2<R> pd = DX[j];
                    contact_term(e, dx, dx1, r0, r1, xyz(pd.a), xyz(pd.b), sp, fa, Ha, fb, Hb);
                }
            } else {
            int c2 = lane;
            V3<R> r0n(R(0)), r1n(R(0));
            D2<R> pdn;
            bool okn = false;
            if (c2 < nc) {
                const int j = packed_partner(__ldg(cl + c2));
                okn = partner_ok(d, j);
                if (okn) {
                    partner_rel(d, off + c2, j, p0, r0n, r1n);
                    pdn = DX[j];
                }
            }
            while (c2 < nc) {
                const V3<R> r0 = r0n, r1 = r1n;
                const D2<R> pd = pdn;
                const bool ok = okn;
                c2 += T;
                if (c2 < nc) {
                    const int j = packed_partner(__ldg(cl + c2));
                    okn = partner_ok(d, j);
                    if (okn) {
                        partner_rel(d, off + c2, j, p0, r0n, r1n);
                        pdn = DX[j];
                    }
                }
                if (ok) contact_term(e, dx, dx1, r0, r1, xyz(pd.a), xyz(pd.b), sp, fa, Ha, fb, Hb);
            }
            }
        }
    }
    if (T > 1) {
        fa.x = slot_sum<R, T>(fa.x); fa.y = slot_sum<R, T>(fa.y); fa.z = slot_sum<R, T>(fa.z);
        fb.x = slot_sum<R, T>(fb.x); fb.y = slot_sum<R, T>(fb.y); fb.z = slot_sum<R, T>(fb.z);
#pragma unroll
        for (int e = 0; e < 6; e++) {
            Ha.d[e] = slot_sum<R, T>(Ha.d[e]);
            Hb.d[e] = slot_sum<R, T>(Hb.d[e]);
        }
    }
    if (lane == 0) {
        sFb[0][t] = fb.x; sFb[1][t] = fb.y; sFb[2][t] = fb.z;
#pragma unroll
        for (int e = 0; e < 6; e++) sHb[e][t] = Hb.d[e];
        sSL[t] = sl;
    }
    __syncthreads();

    // Vertex solve: own segment + previous segment's endpoint share (cosserat.cu:175-205)
    V3<R> dxn = dx;
    if (valid && t > 0) {
        if (flags & F_HAS_PREV) {
            fa += V3<R>(sFb[0][t - 1], sFb[1][t - 1], sFb[2][t - 1]);
            H3<R> hp;
#pragma unroll
            for (int e = 0; e < 6; e++) hp.d[e] = sHb[e][t - 1];
            Ha.add(hp);
            sl = ymin(sl, sSL[t - 1]);
        }
        if (invMass != R(0)) {
            dxn = dx + spp->accel * solve3(Ha, fa);
            const R l = len(dxn);
            if (l > sl && l > R(0)) dxn *= sl / l;
        }
    }
    if (lane == 0) { sDX[0][t] = dxn.x; sDX[1][t] = dxn.y; sDX[2][t] = dxn.z; }
    const bool core = valid && t >= 1 && t <= CORE;
    __syncthreads();

    // New iterate pair and orientation update of segment k (cosserat.cu:209-253)
    if (core && lane == 0) {
        const V3<R> dxb(sDX[0][t + 1], sDX[1][t + 1], sDX[2][t + 1]);
        D2<R> o;
        o.a = v4(dxn, R(0));
        o.b = v4(k + 1 < n ? dxb : V3<R>(R(0)), R(0));
        d.dx[src ^ 1][k] = o;
        Q<R> qn = q0;
        if (!(flags & F_FIX_ORI) && (flags & F_HAS_NEXT)) {
            V3<R> v = ((p1 - p0) + (dxb - dxn)) * (R(1) / lRest);
            v *= R(-2) * kStretch;
            Q<R> b = qmk(R(0), R(0), R(0), R(0));
            if (flags & F_HAS_PREV) {
                const Q<R> qr = qof(d.qRest[k - 1]);
                const Q<R> qq = qof(QO[k - 1]);
                const R s = qdot(qmul(qinv(qq), q0), qr) > R(0) ? R(1) : R(-1);
                b = qadd(b, qscale(s, qmul(qq, qr)));
            }
            if (flags & F_HAS_NEXT_ORI) {
                const Q<R> qr = qof(d.qRest[k]);
                const Q<R> qq = qof(QO[k + 1]);
                const R s = qdot(qmul(qinv(q0), qq), qr) > R(0) ? R(1) : R(-1);
                b = qadd(b, qscale(s, qmul(qq, qinv(qr))));
            }
            // A single-segment yarn has no bending neighbours (b = 0): the closed form is
            // 0/0 there (the reference produces NaN); keep the orientation instead.
            const R bl = qlen(b);
            if (bl > R(0)) {
                const R lambda = len(v) + bl;
                const Q<R> vb1 = qmul(qmul(qmk(v, R(0)), b), qmk(R(1), R(0), R(0), R(0)));
                qn = qnormalize(qadd(vb1, qscale(lambda, b)));
            }
        }
        d.q[src ^ 1][k] = v4of(qn);
    }
}

// ---------------------------------------------------------------------------------------
// Load-balanced kernel (one lane per vertex), the default.  The contact lists of a block's B
// segments are consecutive in the packed layout; the block works through them in two stages:
//   * every warp tests a run of the contacts, one per lane, for being certainly out of range.
//     More than half of the listed contacts are farther apart than the barrier reaches (the lists
//     hold every pair within the detection radius); such a contact contributes exactly zero.
//     No point pair of two segments can be closer than their distance at the start of the
//     substep (from the list pass) less the largest relative displacement of their end points,
//     so a contact with dist - max |dx_a - dx_b| > 2 radius + barrierThickness, by a margin for the
//     rounding of the distances (contact_step_limit), needs no closest points.  The bound is nearly tight, since neighbours move together: 56 % of the
//     entries certified where 59 % are out of range (pile of 65,536 vertices, 12.4 contacts a
//     segment), 59 of 65 % (uneven batch after 3 frames), 99 of 99 % (bundle of parallel yarns);
//   * the others, queued in order, are evaluated NT at a time, one per thread; contributions go
//     through shared memory and the owning thread adds its own in list order.
// Both stages run on full warps, whatever the lengths of the lists, and a warp's long lists are
// shared by the block.  Skipping a contact without the queue would save nothing, since nearly
// every warp holds one in range.  Results are bit for bit those of evaluating every contact.  The
// vertex's own terms are loaded and added after the loop (their inputs are not live across it).
// Bound by issue (53 % of the slots) and by the latency of the gathers, at 24 warps an SM; with 32
// (64 registers, spilled) the large batch takes 6.43 ms per substep and the small scenes 10-20 %
// longer than with 24.  Measured, 8 launches, every contact evaluated -> now: 8.4M vertices with
// 3.2 contacts 7.91 -> 6.69 ms, bundle of 100,352 vertices with 13.7 contacts 336 -> 171 us, pile
// of 65,792 with 11.5 contacts 324 -> 285 us, of 262,144 with 10.6 contacts 898 -> 925 us.
template <typename R>
__device__ __forceinline__ R rel2(const V4<R>& a, const V4<R>& b) {
    const R x = a.x - b.x, y = a.y - b.y, z = a.z - b.z;
    return x * x + y * y + z * z;
}

template <typename R, int B, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) k_iter_bal(Dev<R> d, int src) {
    constexpr int CORE = B - 2;
    constexpr int NW = NT / 32;
    constexpr int SPAN = 256;  // contacts a warp tests before the queue is worked off
    static_assert(B <= 256 && B <= NT, "the owner byte of a packed contact names a slot of the block");
    after_previous_kernel();
    const unsigned FULL = 0xffffffffu;
    const int t = threadIdx.x, lane = t & 31, wp = t >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const int kb = blockIdx.x * CORE - 1, k = kb + t;
    const int n = d.n;
    const bool owns = B == NT || t < B;  // the others only help with the contacts
    const bool valid = owns && (k >= 0) && (k < n);
    const D2<R>* __restrict__ DX = d.dx[src];
    const V4<R>* __restrict__ QO = d.q[src];

    __shared__ V4<R> sA[B], sB[B];  // (dx, e.x) and (dx1, e.y) of each slot's segment, e = p1 - p0
    __shared__ R sEz[B];
    __shared__ int sScene[B];
    // contributions of NT contacts in 16-byte groups: (fa, fb.x) (fb.yz, Ha0-1) (Ha2-5) (Hb0-3),
    // then (Hb4-5)
    __shared__ V4<R> sCon4[4][NT];
    __shared__ R2<R> sCon2[NT];
    __shared__ int sQueue[NW][SPAN];  // contacts to evaluate: place in the block's lists | owner << 16
    __shared__ int sCount[2][NW];  // (two, so that a warp ahead of the others overwrites none that is still read)
    __shared__ short sFirst[B], sEnd[B];  // each owner's entries among those evaluated

    V3<R> fa(R(0)), fb(R(0));
    H3<R> Ha, Hb;
    Ha.zero(); Hb.zero();
    int sc = 0;
    bool sound = true;
    const unsigned base = d.csrOff[max(kb, 0)];
    int total = (int)(d.csrOff[min(kb + B, n)] - base);
    if (valid) {
        // inputs of the vertex's own terms, used after the contact loop
        prefetch_l1(d.vel + k);
        prefetch_l1(QO + k);
        prefetch_l1(d.qRest + k);
        prefetch_l1(d.stepLim + k);
        const unsigned off = d.csrOff[k], end = d.csrOff[k + 1];
        const V4<R> P = d.pos[k];
        const V4<R> P1 = d.pos[min(k + 1, n - 1)];
        const D2<R> own = DX[k];
        sc = scene_of(d.vp[k].flags);
        V4<R> w;
        w.x = own.a.x; w.y = own.a.y; w.z = own.a.z; w.w = P1.x - P.x; sA[t] = w;
        w.x = own.b.x; w.y = own.b.y; w.z = own.b.z; w.w = P1.y - P.y; sB[t] = w;
        sEz[t] = P1.z - P.z;
        sScene[t] = sc;
        sound = end >= off && end - off <= (unsigned)MAX_COLS && end <= d.csrCap;
    }
    if (owns) {
        sFirst[t] = 0;
        sEnd[t] = 0;
    }
    // ranges the packed arrays cannot hold (only after a list pass that reported a failure): the
    // block's lists read as empty
    if (!__syncthreads_and(sound)) total = 0;

    int turn = 0;
    for (int f00 = 0; f00 < total; f00 += NW * SPAN, turn ^= 1) {
        // this warp's contacts: a whole number of steps of 32
        const int share = (min(total - f00, NW * SPAN) + 32 * NW - 1) / (32 * NW) * 32;
        const int fBeg = f00 + wp * share, fEnd = min(fBeg + share, total);
        {
            int qn = 0;  // queued contacts (identical in every lane)
            // A lane's contact is looked up two steps ahead (partner id, owner, squared room) and
            // its partner's iterate loaded one step ahead.
            int j1 = -1, j2 = -1, s1 = 0, s2 = 0;
            R room1 = R(0), room2 = R(0);
            D2<R> p1;
            auto look = [&](int f) {
                j2 = -1;
                if (f < fEnd) {
                    const unsigned g = base + (unsigned)f;
                    const unsigned e = __ldg(d.csrCols + g);
                    j2 = packed_partner(e);
                    s2 = packed_owner(e);
                    room2 = g < d.relCap ? d.relD[g] : R(-1);
                    if (!partner_ok(d, j2)) j2 = -1;
                }
            };
            look(fBeg + lane);
            j1 = j2; s1 = s2; room1 = room2;
            if (j1 >= 0) p1 = DX[j1];
            look(fBeg + 32 + lane);
            for (int f = fBeg + lane; f - lane < fEnd; f += 32) {
                const int j = j1, s = (s1 - kb) & 255;
                const R room = room1;
                const D2<R> pd = p1;
                j1 = j2; s1 = s2; room1 = room2;
                if (j1 >= 0) p1 = DX[j1];
                look(f + 64);
                bool live = false;
                if (j >= 0) {
                    const V4<R> A = sA[s], Bq = sB[s];
                    // room is negative for a contact in range from the start; a comparison with
                    // something that is not a number keeps the contact
                    live = !(rel2(A, pd.a) < room && rel2(A, pd.b) < room && rel2(Bq, pd.a) < room &&
                             rel2(Bq, pd.b) < room);
                }
                const unsigned lives = __ballot_sync(FULL, live);
                if (live) {
                    sQueue[wp][qn + __popc(lives & lt)] = f | s << 16;
                    const unsigned g = base + (unsigned)f;
                    if (g < d.relCap) {
                        prefetch_l1(d.relA + g);
                        prefetch_l1(d.relB + g);
                    }
                }
                qn += __popc(lives);
            }
            if (lane == 0) sCount[turn][wp] = qn;
        }
        __syncthreads();
        int before[NW + 1];
        before[0] = 0;
#pragma unroll
        for (int w = 0; w < NW; w++) before[w + 1] = before[w] + sCount[turn][w];
        const int lives = before[NW];
        auto queued = [&](int i) {  // entry i of the warps' queues, one after the other
            int w = 0, o = 0;
#pragma unroll
            for (int v = 1; v < NW; v++)
                if (i >= before[v]) {
                    w = v;
                    o = before[v];
                }
            return sQueue[w][i - o];
        };
        for (int i0 = 0; i0 < lives; i0 += NT) {
            const int i = i0 + t;
            V3<R> cfa(R(0)), cfb(R(0));
            H3<R> cHa, cHb;
            cHa.zero(); cHb.zero();
            if (i < lives) {
                const int e = queued(i);
                const int s = e >> 16;
                if (t == 0 || queued(i - 1) >> 16 != s) sFirst[s] = (short)t;
                if (t == NT - 1 || i + 1 == lives || queued(i + 1) >> 16 != s) sEnd[s] = (short)(t + 1);
                const unsigned g = base + (unsigned)(e & 0xffff);
                const int j = packed_partner(__ldg(d.csrCols + g));
                const D2<R> pd = DX[j];
                const V4<R> A = sA[s], Bq = sB[s];
                V3<R> r0, r1;
                if (g < d.relCap) {
                    const V4<R> ra = d.relA[g];
                    const R2<R> rb = d.relB[g];
                    r0 = V3<R>(ra.x, ra.y, ra.z);
                    r1 = V3<R>(ra.w, rb.x, rb.y);
                } else {
                    const V3<R> p0 = xyz(d.pos[kb + s]);
                    r0 = xyz(d.pos[j]) - p0;
                    r1 = xyz(d.pos[j + 1]) - p0;
                }
                contact_term(V3<R>(A.w, Bq.w, sEz[s]), xyz(A), xyz(Bq), r0, r1, xyz(pd.a), xyz(pd.b), d.sp[sScene[s]],
                             cfa, cHa, cfb, cHb);
                V4<R> w;
                w.x = cfa.x; w.y = cfa.y; w.z = cfa.z; w.w = cfb.x; sCon4[0][t] = w;
                w.x = cfb.y; w.y = cfb.z; w.z = cHa.d[0]; w.w = cHa.d[1]; sCon4[1][t] = w;
                w.x = cHa.d[2]; w.y = cHa.d[3]; w.z = cHa.d[4]; w.w = cHa.d[5]; sCon4[2][t] = w;
                w.x = cHb.d[0]; w.y = cHb.d[1]; w.z = cHb.d[2]; w.w = cHb.d[3]; sCon4[3][t] = w;
                R2<R> w2;
                w2.x = cHb.d[4]; w2.y = cHb.d[5];
                sCon2[t] = w2;
            }
            __syncthreads();
            if (owns) {
                const int g1 = sEnd[t];
                for (int g = sFirst[t]; g < g1; g++) {
                    const V4<R> c0 = sCon4[0][g], c1 = sCon4[1][g], c2 = sCon4[2][g], c3 = sCon4[3][g];
                    const R2<R> c4 = sCon2[g];
                    fa += V3<R>(c0.x, c0.y, c0.z);
                    fb += V3<R>(c0.w, c1.x, c1.y);
                    Ha.d[0] += c1.z; Ha.d[1] += c1.w;
                    Ha.d[2] += c2.x; Ha.d[3] += c2.y; Ha.d[4] += c2.z; Ha.d[5] += c2.w;
                    Hb.d[0] += c3.x; Hb.d[1] += c3.y; Hb.d[2] += c3.z; Hb.d[3] += c3.w;
                    Hb.d[4] += c4.x; Hb.d[5] += c4.y;
                }
                sFirst[t] = 0;
                sEnd[t] = 0;
            }
            __syncthreads();
        }
    }
    if (!owns) return;
    auto sync_owners = [] {  // a barrier of the owning threads
        if constexpr (B == NT) __syncthreads();
        else if constexpr (B == 32) __syncwarp();
        else asm volatile("bar.sync 1, %0;" ::"n"(B) : "memory");
    };

    // The halo exchange after the loop uses the contributions' memory, viewed as rows of B values.
    R (*rows)[B] = reinterpret_cast<R (*)[B]>(&sCon4[0][0]);
    R (*sFb)[B] = rows;       // rows 0-2
    R (*sHb)[B] = rows + 3;   // rows 3-8
    R* sSL = rows[9];
    R (*sDX)[B] = rows + 10;  // rows 10-12

    // the vertex's own terms (cosserat.cu:40-81)
    R sl = yinf<R>();
    uint32_t flags = 0;
    R invMass = R(0), lRest = R(1), kStretch = R(0);
    V3<R> e(R(0)), dx(R(0));
    Q<R> q0 = qmk(R(0), R(0), R(0), R(1));
    const SceneParams<R>* spp = d.sp;
    if (valid) {
        spp = &d.sp[sc];
        const V4<R> A = sA[t], Bq = sB[t];
        dx = xyz(A);
        e = V3<R>(A.w, Bq.w, sEz[t]);
        add_own_terms(d, k, DX, QO, *spp, xyz(d.pos[k]), e, dx, xyz(Bq), fa, Ha, fb, Hb, flags, invMass, lRest,
                      kStretch, sl, q0);
    }

    sFb[0][t] = fb.x; sFb[1][t] = fb.y; sFb[2][t] = fb.z;
#pragma unroll
    for (int q = 0; q < 6; q++) sHb[q][t] = Hb.d[q];
    sSL[t] = sl;
    sync_owners();

    V3<R> dxn = dx;
    if (valid && t > 0) {
        if (flags & F_HAS_PREV) {
            fa += V3<R>(sFb[0][t - 1], sFb[1][t - 1], sFb[2][t - 1]);
            H3<R> hp;
#pragma unroll
            for (int q = 0; q < 6; q++) hp.d[q] = sHb[q][t - 1];
            Ha.add(hp);
            sl = ymin(sl, sSL[t - 1]);
        }
        if (invMass != R(0)) {
            dxn = dx + spp->accel * solve3(Ha, fa);
            const R l = len(dxn);
            if (l > sl && l > R(0)) dxn *= sl / l;
        }
    }
    sDX[0][t] = dxn.x; sDX[1][t] = dxn.y; sDX[2][t] = dxn.z;
    const bool core = valid && t >= 1 && t <= CORE;
    sync_owners();

    if (core) {
        const V3<R> dxb(sDX[0][t + 1], sDX[1][t + 1], sDX[2][t + 1]);
        D2<R> o;
        o.a = v4(dxn, R(0));
        o.b = v4(k + 1 < n ? dxb : V3<R>(R(0)), R(0));
        d.dx[src ^ 1][k] = o;
        d.q[src ^ 1][k] = v4of(orientation_update(d, k, QO, flags, e, dxn, dxb, lRest, kStretch, q0));
    }
}

// ---------------------------------------------------------------------------------------
// The same iteration without the test: every contact is evaluated, NT at a time, one per thread.
// The better one for large simulations whose listed contacts are mostly in range (settled piles):
// there the test costs more than the few contacts it spares.  72 registers, 7 blocks an SM.  Bound by
// issue and the latency of the gathers.  Measured, us a launch, k_iter_bal against this kernel by the
// share of listed contacts that are in range when a substep starts: 1.0M vertices in 32 scenes, 17 %:
// 100 against 119, 32 %: 119 / 128, 46 %: 142 / 140, 53 %: 164 / 156, 57 %: 180 / 169; 8.4M in 269 scenes,
// 34 %: 943 / 986, 47 %: 1080 / 1047, 55 %: 1207 / 1134; pile of 262,144 vertices, 48 %: 108 / 111, 57 %:
// 107 / 101, 61 %: 104 / 93; pile of 65,792, where the grid is less than a wave, 58 %: 35 / 37.
// Results are the same bit for bit.
template <typename R, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) k_iter_all(Dev<R> d, int src) {
    after_previous_kernel();
    constexpr int B = NT;
    constexpr int CORE = B - 2;
    constexpr int NW = NT / 32;
    const int t = threadIdx.x;
    const int k = blockIdx.x * CORE - 1 + t;
    const int n = d.n;
    const bool valid = (k >= 0) && (k < n);
    const D2<R>* __restrict__ DX = d.dx[src];
    const V4<R>* __restrict__ QO = d.q[src];

    __shared__ R sSeg[12][B];  // p0, e = p1 - p0, dx, dx1 of each slot's segment
    // contributions of one chunk of contacts, double buffered, in 16-byte groups:
    // (fa, fb.x) (fb.yz, Ha0-1) (Ha2-5) (Hb0-3), then (Hb4-5)
    __shared__ V4<R> sCon4[2][4][B];
    __shared__ R2<R> sCon2[2][B];
    __shared__ int sOwn[2][B];     // owning slot of each contact of a chunk (double buffered)
    __shared__ int sOff[B + 1];
    __shared__ int sScene[B];
    __shared__ int sWarp[NW];
    __shared__ unsigned sBase;

    // The contact loop runs first and accumulates from zero; the vertex's own terms (inertia,
    // glue, stretch) are loaded and added after it, so their inputs are not live (in
    // registers) across the loop.
    V3<R> fa(R(0)), fb(R(0));
    H3<R> Ha, Hb;
    Ha.zero(); Hb.zero();
    int nc = 0, sc = 0;
    if (t == 0) sBase = d.csrOff[k < 0 ? 0 : k];  // the block's first packed slot (k < n here)
    {
        V3<R> p0(R(0)), e(R(0)), dx(R(0)), dx1(R(0));
        if (valid) {
            // inputs of the vertex's own terms, used after the contact loop
            prefetch_l1(d.vel + k);
            prefetch_l1(QO + k);
            prefetch_l1(d.qRest + k);
            prefetch_l1(d.stepLim + k);
            const uint32_t fl = d.vp[k].flags;
            sc = scene_of(fl);
            const D2<R> own = DX[k];
            dx = xyz(own.a);
            dx1 = xyz(own.b);
            p0 = xyz(d.pos[k]);
            if (fl & F_HAS_NEXT) {
                e = xyz(d.pos[k + 1]) - p0;
                unsigned off;
                nc = contact_range(d, k, off);
            }
        }
        sSeg[0][t] = p0.x; sSeg[1][t] = p0.y; sSeg[2][t] = p0.z;
        sSeg[3][t] = e.x; sSeg[4][t] = e.y; sSeg[5][t] = e.z;
        sSeg[6][t] = dx.x; sSeg[7][t] = dx.y; sSeg[8][t] = dx.z;
        sSeg[9][t] = dx1.x; sSeg[10][t] = dx1.y; sSeg[11][t] = dx1.z;
        sScene[t] = sc;
    }
    // block exclusive scan of the contact counts (the block's packed slots are base + offset)
    {
        const int lane = t & 31, w = t >> 5;
        int x = nc;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) sWarp[w] = x;
        __syncthreads();
        int wo = 0;
        for (int i = 0; i < w; i++) wo += sWarp[i];
        sOff[t] = wo + x - nc;
        if (t == B - 1) sOff[B] = wo + x;
        __syncthreads();
    }
    int total = sOff[B];
    int myOff = sOff[t];
    const unsigned base = sBase;
    if (base > d.csrCap || d.csrCap - base < (unsigned)total) {  // only a packing the list pass reported as failed
        total = 0;
        myOff = 0;
        nc = 0;
    }
    // Chunks of NT contacts, one per thread.  Each thread writes its own slot index over its
    // contacts of the next chunk before the current chunk's barrier, which publishes it, and
    // the contributions are double buffered: a buffer is written again only after the next
    // chunk's barrier, which every thread reaches after summing it, so each chunk needs one
    // barrier.
    for (int g = myOff; g < min(myOff + nc, NT); g++) sOwn[0][g] = t;
    __syncthreads();
    int buf = 0;
    // The packed contact of this thread is loaded one chunk ahead (after the previous chunk's barrier,
    // before its summation), so a chunk starts with the partner gather; it is unpacked there, since an
    // operation on it here would wait for the load (+5 % on the whole kernel).
    unsigned en = 0;
    if (t < total) en = __ldg(d.csrCols + (base + t));
    for (int b0 = 0; b0 < total; b0 += NT, buf ^= 1) {
        const int f = b0 + t;
        {
            const int nb = b0 + NT;
            const int g1 = min(myOff + nc, nb + NT);
            for (int g = max(myOff, nb); g < g1; g++) sOwn[buf ^ 1][g - nb] = t;
        }
        V3<R> cfa(R(0)), cfb(R(0));
        H3<R> cHa, cHb;
        cHa.zero(); cHb.zero();
        const int j = packed_partner(en);
        if (f < total && partner_ok(d, j)) {
            const int s = sOwn[buf][t];
            const V3<R> sp0(sSeg[0][s], sSeg[1][s], sSeg[2][s]);
            V3<R> r0, r1;
            partner_rel(d, base + f, j, sp0, r0, r1);
            const D2<R> pd = DX[j];
            const V3<R> se(sSeg[3][s], sSeg[4][s], sSeg[5][s]);
            const V3<R> sdx(sSeg[6][s], sSeg[7][s], sSeg[8][s]);
            const V3<R> sdx1(sSeg[9][s], sSeg[10][s], sSeg[11][s]);
            contact_term(se, sdx, sdx1, r0, r1, xyz(pd.a), xyz(pd.b), d.sp[sScene[s]], cfa, cHa, cfb, cHb);
        }
        {
            V4<R> w;
            w.x = cfa.x; w.y = cfa.y; w.z = cfa.z; w.w = cfb.x; sCon4[buf][0][t] = w;
            w.x = cfb.y; w.y = cfb.z; w.z = cHa.d[0]; w.w = cHa.d[1]; sCon4[buf][1][t] = w;
            w.x = cHa.d[2]; w.y = cHa.d[3]; w.z = cHa.d[4]; w.w = cHa.d[5]; sCon4[buf][2][t] = w;
            w.x = cHb.d[0]; w.y = cHb.d[1]; w.z = cHb.d[2]; w.w = cHb.d[3]; sCon4[buf][3][t] = w;
            R2<R> w2;
            w2.x = cHb.d[4]; w2.y = cHb.d[5];
            sCon2[buf][t] = w2;
        }
        __syncthreads();
        {
            // next chunk: partner id, and the staged partner positions into L1
            const int fn = b0 + NT + t;
            if (fn < total) {
                const unsigned g = base + fn;
                en = __ldg(d.csrCols + g);
                if (g < d.relCap) {
                    prefetch_l1(d.relA + g);
                    prefetch_l1(d.relB + g);
                }
            }
        }
        const int f0 = max(myOff, b0), f1 = min(myOff + nc, b0 + NT);
        for (int g = f0; g < f1; g++) {
            const int i = g - b0;
            const V4<R> w0 = sCon4[buf][0][i], w1 = sCon4[buf][1][i], w2 = sCon4[buf][2][i], w3 = sCon4[buf][3][i];
            const R2<R> w4 = sCon2[buf][i];
            fa += V3<R>(w0.x, w0.y, w0.z);
            fb += V3<R>(w0.w, w1.x, w1.y);
            Ha.d[0] += w1.z; Ha.d[1] += w1.w;
            Ha.d[2] += w2.x; Ha.d[3] += w2.y; Ha.d[4] += w2.z; Ha.d[5] += w2.w;
            Hb.d[0] += w3.x; Hb.d[1] += w3.y; Hb.d[2] += w3.z; Hb.d[3] += w3.w;
            Hb.d[4] += w4.x; Hb.d[5] += w4.y;
        }
    }

    // The halo exchange after the loop uses the contribution buffer the last chunk did not
    // use (buf), viewed as 16 rows of B values: every thread finished reading it before the
    // last chunk's barrier.
    R (*rows)[B] = reinterpret_cast<R (*)[B]>(&sCon4[buf][0][0]);
    R (*sFb)[B] = rows;       // rows 0-2
    R (*sHb)[B] = rows + 3;   // rows 3-8
    R* sSL = rows[9];
    R (*sDX)[B] = rows + 10;  // rows 10-12

    // the vertex's own terms (cosserat.cu:40-81)
    R sl = yinf<R>();
    uint32_t flags = 0;
    R invMass = R(0), lRest = R(1), kStretch = R(0);
    const V3<R> p0(sSeg[0][t], sSeg[1][t], sSeg[2][t]);
    const V3<R> e(sSeg[3][t], sSeg[4][t], sSeg[5][t]);
    const V3<R> dx(sSeg[6][t], sSeg[7][t], sSeg[8][t]);
    Q<R> q0 = qmk(R(0), R(0), R(0), R(1));
    const SceneParams<R>* spp = d.sp;
    if (valid) {
        spp = &d.sp[sc];
        add_own_terms(d, k, DX, QO, *spp, p0, e, dx, V3<R>(sSeg[9][t], sSeg[10][t], sSeg[11][t]), fa, Ha, fb, Hb,
                      flags, invMass, lRest, kStretch, sl, q0);
    }

    sFb[0][t] = fb.x; sFb[1][t] = fb.y; sFb[2][t] = fb.z;
#pragma unroll
    for (int q = 0; q < 6; q++) sHb[q][t] = Hb.d[q];
    sSL[t] = sl;
    __syncthreads();

    V3<R> dxn = dx;
    if (valid && t > 0) {
        if (flags & F_HAS_PREV) {
            fa += V3<R>(sFb[0][t - 1], sFb[1][t - 1], sFb[2][t - 1]);
            H3<R> hp;
#pragma unroll
            for (int q = 0; q < 6; q++) hp.d[q] = sHb[q][t - 1];
            Ha.add(hp);
            sl = ymin(sl, sSL[t - 1]);
        }
        if (invMass != R(0)) {
            dxn = dx + spp->accel * solve3(Ha, fa);
            const R l = len(dxn);
            if (l > sl && l > R(0)) dxn *= sl / l;
        }
    }
    sDX[0][t] = dxn.x; sDX[1][t] = dxn.y; sDX[2][t] = dxn.z;
    const bool core = valid && t >= 1 && t <= CORE;
    __syncthreads();

    if (core) {
        const V3<R> dxb(sDX[0][t + 1], sDX[1][t + 1], sDX[2][t + 1]);
        D2<R> o;
        o.a = v4(dxn, R(0));
        o.b = v4(k + 1 < n ? dxb : V3<R>(R(0)), R(0));
        d.dx[src ^ 1][k] = o;
        d.q[src ^ 1][k] = v4of(orientation_update(d, k, QO, flags, e, dxn, dxb, lRest, kStretch, q0));
    }
}

// ---------------------------------------------------------------------------------------
// The same iteration for small simulations, where a launch lasts as long as one block's chain of
// dependent steps (some 10k cycles) and most of the chip's issue slots are free.  A block has 32
// slots: warp 0 owns them, the other warps work on the contacts in the same two stages.  While they
// evaluate, the owners form the costly parts of their own terms and the bending gradients, which
// k_iter_bal does after the sums; halo values pass between lanes instead of shared memory.  Every sum
// has k_iter_bal's order and terms, and the parts formed early are chosen so that the compiler fuses
// the rest alike: the results are the same bit for bit.
// Needs 128 registers (FP64 242): at 80, where six blocks of 128 threads fit an SM, 430 bytes spill and
// the launch takes 6 to 20 % longer than k_iter_bal's.  Measured, us per iteration within a substep, k_iter_bal with
// 32 slots -> this kernel, swatches of 780 / 1,949 / 4,032 / 7,900 vertices: 6.2 / 6.2 / 6.4 / 6.7 ->
// 5.1 / 5.4 / 5.4 / 5.6; FP64 build, 780 / 1,949 / 4,032 vertices: 7.2 / 7.0 / 7.6 -> 6.1 / 6.0 / 6.4.
// 192 and 160 threads (112, 96 registers) gain nothing, 384 threads no more than 256.
template <typename R, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) k_iter_small(Dev<R> d, int src) {
    after_previous_kernel();
    constexpr int CORE = 30;
    constexpr int HELP = NT - 32, HW = HELP / 32;
    constexpr int STEPS = 2, SPAN = 32 * STEPS;  // contacts a warp tests before the queue is worked off
    const unsigned FULL = 0xffffffffu;
    const int t = threadIdx.x, lane = t & 31, h = t - 32, wp = h >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const bool owns = t < 32;
    const int kb = blockIdx.x * CORE - 1, k = kb + lane;
    const int n = d.n;
    const bool valid = owns && k >= 0 && k < n;
    const D2<R>* __restrict__ DX = d.dx[src];
    const V4<R>* __restrict__ QO = d.q[src];

    __shared__ V4<R> sA[32], sB[32];  // (dx, e.x) and (dx1, e.y) of each slot's segment, e = p1 - p0
    __shared__ R sEz[32];
    __shared__ int sScene[32];
    __shared__ V4<R> sCon4[4][HELP];  // contributions, grouped as in k_iter_bal
    __shared__ R2<R> sCon2[HELP];
    __shared__ int sQueue[HW][SPAN];  // contacts to evaluate: place in the block's lists | owner << 16
    __shared__ int sCount[2][HW];
    __shared__ short sFirst[32], sEnd[32];  // each owner's entries among those evaluated

    const unsigned base = d.csrOff[max(kb, 0)];
    int total = (int)(d.csrOff[min(kb + 32, n)] - base);
    int sc = 0;
    bool sound = true;
    V3<R> p0(R(0)), e(R(0)), dx(R(0)), dx1(R(0));
    int fBeg = 0, fEnd = 0;  // a helper warp's contacts
    int j[STEPS], s[STEPS];
    R room[STEPS];
    D2<R> pd[STEPS];
    auto load = [&](int f00) {
        const int share = (min(total - f00, HW * SPAN) + 32 * HW - 1) / (32 * HW) * 32;
        fBeg = f00 + wp * share;
        fEnd = min(fBeg + share, total);
#pragma unroll
        for (int q = 0; q < STEPS; q++) {
            const int f = fBeg + 32 * q + lane;
            const unsigned g = base + (unsigned)f;
            j[q] = -1;
            if (f < fEnd && g < d.csrCap) {
                const unsigned e = __ldg(d.csrCols + g);
                j[q] = packed_partner(e);
                s[q] = (packed_owner(e) - kb) & 31;
                room[q] = g < d.relCap ? d.relD[g] : R(-1);
            }
        }
#pragma unroll
        for (int q = 0; q < STEPS; q++) {
            if (!partner_ok(d, j[q])) j[q] = -1;
            if (j[q] >= 0) pd[q] = DX[j[q]];
        }
    };
    if (valid) {
        // inputs of the vertex's own terms, used later
        prefetch_l1(d.vel + k);
        prefetch_l1(QO + k);
        prefetch_l1(d.qRest + k);
        prefetch_l1(d.stepLim + k);
        const unsigned off = d.csrOff[k], end = d.csrOff[k + 1];
        const V4<R> P = d.pos[k];
        const V4<R> P1 = d.pos[min(k + 1, n - 1)];
        const D2<R> own = DX[k];
        sc = scene_of(d.vp[k].flags);
        p0 = xyz(P);
        e = xyz(P1) - p0;
        dx = xyz(own.a);
        dx1 = xyz(own.b);
        sA[lane] = v4(dx, e.x);
        sB[lane] = v4(dx1, e.y);
        sEz[lane] = e.z;
        sScene[lane] = sc;
        sound = end >= off && end - off <= (unsigned)MAX_COLS && end <= d.csrCap;
    } else if (!owns) {
        load(0);
    }
    if (owns) {
        sFirst[lane] = 0;
        sEnd[lane] = 0;
    }
    if (!__syncthreads_and(sound)) total = 0;  // as in k_iter_bal

    V3<R> fa(R(0)), fb(R(0));
    H3<R> Ha, Hb;
    Ha.zero(); Hb.zero();
    OwnParts<R> w;
    Q<R> bend = qmk(R(0), R(0), R(0), R(0));
    bool prepared = false;
    auto prepare = [&] {
        prepared = true;
        if (!valid) return;
        w = own_parts(d, k, QO, d.sp[sc]);
        const uint32_t fl = d.vp[k].flags;
        if (turns(fl)) bend = bending_gradient(d, k, QO, fl, w.q0);
    };
    int turn = 0;
    for (int f00 = 0; f00 < total; f00 += HW * SPAN, turn ^= 1) {
        if (!owns) {
            int qn = 0;  // queued contacts (identical in every lane)
#pragma unroll
            for (int q = 0; q < STEPS; q++) {
                const int f = fBeg + 32 * q + lane;
                bool live = false;
                if (j[q] >= 0) {
                    const V4<R> A = sA[s[q]], Bq = sB[s[q]];
                    live = !(rel2(A, pd[q].a) < room[q] && rel2(A, pd[q].b) < room[q] && rel2(Bq, pd[q].a) < room[q] &&
                             rel2(Bq, pd[q].b) < room[q]);
                }
                const unsigned lives = __ballot_sync(FULL, live);
                if (live) {
                    sQueue[wp][qn + __popc(lives & lt)] = f | s[q] << 16;
                    const unsigned g = base + (unsigned)f;
                    if (g < d.relCap) {
                        prefetch_l1(d.relA + g);
                        prefetch_l1(d.relB + g);
                    }
                }
                qn += __popc(lives);
            }
            if (lane == 0) sCount[turn][wp] = qn;
        }
        __syncthreads();
        int before[HW + 1];
        before[0] = 0;
#pragma unroll
        for (int v = 0; v < HW; v++) before[v + 1] = before[v] + sCount[turn][v];
        const int lives = before[HW];
        auto queued = [&](int i) {  // entry i of the warps' queues, one after the other
            int v = 0, o = 0;
#pragma unroll
            for (int u = 1; u < HW; u++)
                if (i >= before[u]) {
                    v = u;
                    o = before[u];
                }
            return sQueue[v][i - o];
        };
        for (int i0 = 0; i0 < lives; i0 += HELP) {
            const int i = i0 + h;
            if (owns) {
                if (!prepared) prepare();
            } else if (i < lives) {
                const int en = queued(i);
                const int so = en >> 16;
                if (h == 0 || queued(i - 1) >> 16 != so) sFirst[so] = (short)h;
                if (h == HELP - 1 || i + 1 == lives || queued(i + 1) >> 16 != so) sEnd[so] = (short)(h + 1);
                const unsigned g = base + (unsigned)(en & 0xffff);
                const int jo = packed_partner(__ldg(d.csrCols + g));
                const D2<R> po = DX[jo];
                const V4<R> A = sA[so], Bq = sB[so];
                V3<R> r0, r1;
                if (g < d.relCap) {
                    const V4<R> ra = d.relA[g];
                    const R2<R> rb = d.relB[g];
                    r0 = V3<R>(ra.x, ra.y, ra.z);
                    r1 = V3<R>(ra.w, rb.x, rb.y);
                } else {
                    const V3<R> a0 = xyz(d.pos[kb + so]);
                    r0 = xyz(d.pos[jo]) - a0;
                    r1 = xyz(d.pos[jo + 1]) - a0;
                }
                V3<R> cfa(R(0)), cfb(R(0));
                H3<R> cHa, cHb;
                cHa.zero(); cHb.zero();
                contact_term(V3<R>(A.w, Bq.w, sEz[so]), xyz(A), xyz(Bq), r0, r1, xyz(po.a), xyz(po.b), d.sp[sScene[so]],
                             cfa, cHa, cfb, cHb);
                V4<R> c;
                c.x = cfa.x; c.y = cfa.y; c.z = cfa.z; c.w = cfb.x; sCon4[0][h] = c;
                c.x = cfb.y; c.y = cfb.z; c.z = cHa.d[0]; c.w = cHa.d[1]; sCon4[1][h] = c;
                c.x = cHa.d[2]; c.y = cHa.d[3]; c.z = cHa.d[4]; c.w = cHa.d[5]; sCon4[2][h] = c;
                c.x = cHb.d[0]; c.y = cHb.d[1]; c.z = cHb.d[2]; c.w = cHb.d[3]; sCon4[3][h] = c;
                R2<R> c2;
                c2.x = cHb.d[4]; c2.y = cHb.d[5];
                sCon2[h] = c2;
            }
            __syncthreads();
            if (owns) {
                const int g1 = sEnd[lane];
                for (int g = sFirst[lane]; g < g1; g++) {
                    const V4<R> c0 = sCon4[0][g], c1 = sCon4[1][g], c2 = sCon4[2][g], c3 = sCon4[3][g];
                    const R2<R> c4 = sCon2[g];
                    fa += V3<R>(c0.x, c0.y, c0.z);
                    fb += V3<R>(c0.w, c1.x, c1.y);
                    Ha.d[0] += c1.z; Ha.d[1] += c1.w;
                    Ha.d[2] += c2.x; Ha.d[3] += c2.y; Ha.d[4] += c2.z; Ha.d[5] += c2.w;
                    Hb.d[0] += c3.x; Hb.d[1] += c3.y; Hb.d[2] += c3.z; Hb.d[3] += c3.w;
                    Hb.d[4] += c4.x; Hb.d[5] += c4.y;
                }
                sFirst[lane] = 0;
                sEnd[lane] = 0;
            }
            if (i0 + HELP < lives || f00 + HW * SPAN < total) __syncthreads();
        }
        if (!owns && f00 + HW * SPAN < total) load(f00 + HW * SPAN);
    }
    if (!owns) return;
    if (!prepared) prepare();
    uint32_t flags = 0;
    R invMass = R(0), lRest = R(1), kStretch = R(0), sl = yinf<R>();
    Q<R> q0 = qmk(R(0), R(0), R(0), R(1));
    if (valid)
        add_own_terms(d, k, DX, QO, d.sp[sc], p0, e, dx, dx1, fa, Ha, fb, Hb, flags, invMass, lRest, kStretch, sl, q0,
                      &w);

    // the previous segment's shares (cosserat.cu:175-205)
    V3<R> pf(__shfl_up_sync(FULL, fb.x, 1), __shfl_up_sync(FULL, fb.y, 1), __shfl_up_sync(FULL, fb.z, 1));
    H3<R> ph;
#pragma unroll
    for (int q = 0; q < 6; q++) ph.d[q] = __shfl_up_sync(FULL, Hb.d[q], 1);
    const R psl = __shfl_up_sync(FULL, sl, 1);
    V3<R> dxn = dx;
    if (valid && lane > 0) {
        if (flags & F_HAS_PREV) {
            fa += pf;
            Ha.add(ph);
            sl = ymin(sl, psl);
        }
        if (invMass != R(0)) {
            dxn = dx + d.sp[sc].accel * solve3(Ha, fa);
            const R l = len(dxn);
            if (l > sl && l > R(0)) dxn *= sl / l;
        }
    }
    const V3<R> dxb(__shfl_down_sync(FULL, dxn.x, 1), __shfl_down_sync(FULL, dxn.y, 1), __shfl_down_sync(FULL, dxn.z, 1));
    if (valid && lane >= 1 && lane <= CORE) {
        D2<R> o;
        o.a = v4(dxn, R(0));
        o.b = v4(k + 1 < n ? dxb : V3<R>(R(0)), R(0));
        d.dx[src ^ 1][k] = o;
        d.q[src ^ 1][k] = v4of(turns(flags) ? turned(q0, bend, e, dxn, dxb, w.invl, kStretch) : q0);
    }
}

// ---------------------------------------------------------------------------------------
template <typename R>
void launch_init(const Dev<R>& d, bool clearLists, cudaStream_t s) {
    if (d.n <= 0) return;
    launch_dependent(k_init<R>, (d.n + 255) / 256, 256, s, d, clearLists ? 1 : 0);
}

template <typename R>
void launch_end(const Dev<R>& d, int finalBuf, bool copyQ, bool kahan, cudaStream_t s) {
    if (d.n <= 0) return;
    launch_dependent(k_end<R>, (d.n + 255) / 256, 256, s, d, finalBuf, copyQ ? 1 : 0, kahan ? 1 : 0);
}

// Newton iteration launch shapes: NT threads per block, T lanes per vertex, pipelined or not;
// lanes = 0 selects the load-balanced kernel (one lane per vertex, flattened contact lists; pipe
// makes no difference to it).
template <typename R>
void launch_iter(const Dev<R>& d, int srcBuf, int threads, int lanes, int pipe, cudaStream_t s) {
    if (d.n <= 0) return;
#define YB_ITER(NT, T, MINB, P) \
    k_iter<R, NT, T, MINB, P><<<(d.n + (NT / T) - 3) / ((NT / T) - 2), NT, 0, s>>>(d, srcBuf)
    if (lanes == 0) {
        // Load-balanced kernels, chosen by newton_kernel().  A block of 128 slots fills the chip from about
        // 112k vertices on (6 blocks of 126 vertices on 148 SMs).  Below, a launch lasts as long as one
        // block's chain of steps, so small blocks of 32 slots get 3 or 7 warps that only help with the
        // contacts, while the grid still is one wave.  Us per substep of whole advances, 32 slots with
        // 128 threads / with 256 / 128 slots: swatches of 13,580, 19,400 and 25,220 vertices 116 / 134 / 152,
        // 136 / 156 / 197 and 141 / 165 / 212, piles of 14,000 and 26,000 173 / 187 / 261 and 231 / 248 / 305.
        // (Past a wave it would still gain for a while: 141 against 216 at 29,100, 174 against 232 at 48,500, 235
        // against 235 at 77,600; the line does not use that yet.)  8 launches, 256 threads against 128: 69
        // and 69 us at 1,949, 38 and 43 at 12,827.  FP64 build, 32 slots with 128 threads against 128 slots:
        // 147 / 186 us a substep at 13,580, 215 / 269 at 29,100, 294 / 296 at 48,500.
        // k_iter_small wins while its blocks, two to an SM (FP64: one) for their registers, are one
        // wave; past that its second wave costs more: 6.9 against 9.7 us an iteration at 11,875
        // vertices, FP64 8.0 against 11.1 at 7,900.  The results are the same bit for bit.
        // A grid of 128 slots of at most one wave is launched the plain way: set up while the one before
        // runs, its blocks would land on the SMs with the most room left instead of evenly.  Us per substep,
        // plain / dependent: 216 / 228 at 29,100, 232 / 247 at 48,500, 237 / 261 at 77,600, pile of 105,000 753 /
        // 748.  Elsewhere the early set-up gains: 67 -> 59 us at 1,949, 842 -> 827 us at 1.0M.  The FP64
        // build has the plain way throughout: 238 / 246 at 19,400, 269 / 285 at 29,100, 296 / 298 at 48,500, pile of
        // 200,000 1320 / 1317, of 1.0M 5897 / 5877.
        const size_t small = (d.n + 29) / 30, large = (d.n + 125) / 126;
        constexpr bool F32 = sizeof(R) == 4;
        switch (newton_kernel(d)) {
            case NEWTON_SMALL:
                launch_dependent(k_iter_small<R, 256, F32 ? 2 : 1>, small, 256, s, d, srcBuf);
                break;
            case NEWTON_32_WIDE:
                if constexpr (F32) launch_dependent(k_iter_bal<R, 32, 256, 3>, small, 256, s, d, srcBuf);
                break;
            case NEWTON_32:
                launch_dependent(k_iter_bal<R, 32, 128, F32 ? 6 : 3>, small, 128, s, d, srcBuf);
                break;
            case NEWTON_128_PLAIN:
                k_iter_bal<R, 128, 128, F32 ? 6 : 3><<<large, 128, 0, s>>>(d, srcBuf);
                break;
            case NEWTON_128:
                if constexpr (F32) launch_dependent(k_iter_bal<R, 128, 128, 6>, large, 128, s, d, srcBuf);
                break;
            case NEWTON_ALL:
                if constexpr (F32) launch_dependent(k_iter_all<R, 128, 7>, large, 128, s, d, srcBuf);
                break;
            case NEWTON_LANES: break;
        }
    } else if (pipe) {
        if (lanes == 4) YB_ITER(256, 4, 2, true);
        else if (threads == 128) YB_ITER(128, 1, 4, true);
        else YB_ITER(256, 1, 2, true);
    } else if (lanes == 2) {
        YB_ITER(256, 2, 3, false);
    } else if (lanes == 4) {
        if (threads == 512) YB_ITER(512, 4, 2, false); else YB_ITER(256, 4, 3, false);
    } else if (lanes == 8) {
        if (threads == 512) YB_ITER(512, 8, 2, false); else YB_ITER(256, 8, 3, false);
    } else {
        if (threads == 128) YB_ITER(128, 1, 6, false); else YB_ITER(256, 1, 2, false);
    }
#undef YB_ITER
}

template void launch_init<float>(const Dev<float>&, bool, cudaStream_t);
template void launch_init<double>(const Dev<double>&, bool, cudaStream_t);
template void launch_end<float>(const Dev<float>&, int, bool, bool, cudaStream_t);
template void launch_end<double>(const Dev<double>&, int, bool, bool, cudaStream_t);
template void launch_iter<float>(const Dev<float>&, int, int, int, int, cudaStream_t);
template void launch_iter<double>(const Dev<double>&, int, int, int, int, cudaStream_t);

}  // namespace yb
