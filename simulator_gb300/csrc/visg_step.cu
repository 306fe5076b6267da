// visg_step.cu — the fused cloth step and the first-hit query.
//
// k_step is the reference's `verlet` kernel (src/verlet.cu:129-161) rebuilt for
// GB300: one thread per vertex, persistent CTAs walking a tile table (a tile is
// BLOCK consecutive vertices of one garment, so one launch covers any number of
// garments of uneven size) or persistent warps walking slices of 32 vertices, state
// records in two 16-byte halves (one float4 load per spring neighbour when spring damping
// is zero, two otherwise), springs of all lists merged into one sliced-ELL table of 8-byte
// entries (optionally staged per slice in shared memory by TMA bulk copies while the warp
// finishes the slice before) summed list by list with the list's stiffness uniform across the loop, the previous
// contact normal read only for vertices that had a contact, and the collision
// (collision_response_projection, verlet.cu:24-50) fused behind a warp vote on the
// body's root box.  Arithmetic follows the reference operation by operation with
// explicit round-to-nearest intrinsics:
//   v  = (x - xo) / dt
//   F  = g*m + v*damp;  F += sum_list (sum_entry spring);  F -= (n_prev.F) n_prev
//   spring = (-k (|d| - L0) + kd (dv.d)/|d|) * normalize(d),  d = x - x_j + FLT_EPSILON
//   x' = (x + x - xo) + (F/m*dt)*dt       (gamma == 1, verlet.cu:155)
//   x' = (x + gamma (x - xo)) + (F/m*dt)*dt  (damped Verlet)
//   first-hit leaf (cudaBRT.cu:239-285) -> plane test (primitive.cu:110-125)
//   -> x' += |dist| n, xo' = x', n_prev' = n; else n_prev' = 0
#include <cuda_runtime.h>
#include <limits.h>
#include <stdint.h>

#include <map>
#include <mutex>

#include "visg_internal.cuh"
#include "visg_launch.cuh"

namespace visg {

namespace {

constexpr float kFltEpsilon = 1.1920928955078125e-07f;  // FLT_EPSILON
constexpr int kStack = 32;  // > 30 = the depth bound of a radix tree over distinct 30-bit codes

__device__ __forceinline__ bool in_box(f3 p, float4 lo, float4 hi) {  // BBox::intersect, inclusive
    return (p.x >= lo.x && p.x <= hi.x) && (p.y >= lo.y && p.y <= hi.y) && (p.z >= lo.z && p.z <= hi.z);
}

// the larger of two floats, NaN if either is (fmaxf drops a NaN)
__device__ __forceinline__ float max_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

// Upper bound of max_axis |a - b| (each difference rounded up); NaN, which no margin covers,
// if a coordinate is.
__device__ __forceinline__ float disp_bound(f3 a, f3 b) {
    const float dx = max_nan(__fsub_ru(a.x, b.x), __fsub_ru(b.x, a.x));
    const float dy = max_nan(__fsub_ru(a.y, b.y), __fsub_ru(b.y, a.y));
    const float dz = max_nan(__fsub_ru(a.z, b.z), __fsub_ru(b.z, a.z));
    return max_nan(dx, max_nan(dy, dz));
}

// Lower bounds (differences rounded down) of the L-infinity distance p can move
// before the closed-box test (BBox::intersect) changes its answer: outside the box,
// the largest per-axis gap; inside, the distance to the nearest face.
// A rounded-down difference has the sign of the exact one (a difference of two floats is zero
// only if they are equal), so a point is in the closed box exactly when its gap is not
// positive, if neither has a NaN.  A tree's boxes have none (build_chunk).
__device__ __forceinline__ float box_gap(f3 p, float4 lo, float4 hi) {
    return fmaxf(fmaxf(fmaxf(__fsub_rd(lo.x, p.x), __fsub_rd(p.x, hi.x)), fmaxf(__fsub_rd(lo.y, p.y), __fsub_rd(p.y, hi.y))),
                 fmaxf(__fsub_rd(lo.z, p.z), __fsub_rd(p.z, hi.z)));
}
__device__ __forceinline__ float box_inner(f3 p, float4 lo, float4 hi) {
    return fminf(fminf(fminf(__fsub_rd(p.x, lo.x), __fsub_rd(hi.x, p.x)), fminf(__fsub_rd(p.y, lo.y), __fsub_rd(hi.y, p.y))),
                 fminf(__fsub_rd(p.z, lo.z), __fsub_rd(hi.z, p.z)));
}

// D_BVH::intersect semantics: children tested pairwise; an overlapping leaf child is
// returned before any descent (A before B); both internal -> descend A, push B.
// The answer is therefore the first leaf, in a fixed order of the tree's leaves,
// whose box contains p (a node's box contains its children's).  A depth-first walk
// visits every internal node at most once, so `budget` (the number of internal
// nodes) bounds the loop even on a corrupted tree.
// m receives a distance a point may move from p and keep the answer:
// every leaf before the answer lies under a box the walk rejected (min of their
// gaps), and the answer's own box must keep containing it (its inner distance).
// A walk is one chain of dependent loads (285 cycles each when they miss the L1) and of
// what is computed between them, which with a branch per outcome took longer than the
// load: the lanes of a warp part at every visit.  So a visit has no branch but the loop's:
// one signed gap per box serves the test and the margin, the next link is selected (a
// leaf's or the empty stack's is negative and ends the walk), and the stack is written and
// read at every visit, used or not, with its top in a register.
// p has no NaN (query_margin sees to it).
__device__ __forceinline__ int first_hit(const Node* nodes, int node, int budget, f3 p, int* err,
                                         float& m) {
    constexpr int kEmpty = INT_MIN;
    const float inf = __int_as_float(0x7f800000);
    int stack[kStack];
    int sp = 0, top = kEmpty;
    f4x2 a, b;
    bool hit_a;
    do {
        a = ld8(&nodes[node].a_lo);
        b = ld8(&nodes[node].b_lo);
        stack[sp] = top;
        const int below = stack[max(sp - 1, 0)];
        const int la = __float_as_int(a.a.w), lb = __float_as_int(b.a.w);
        const float ga = box_gap(p, a.a, a.b), gb = box_gap(p, b.a, b.b);
        const bool in_a = !(ga > 0.0f), in_b = !(gb > 0.0f);
        hit_a = in_a && la < 0;
        const bool hit_b = in_b && lb < 0 && !hit_a;
        m = fminf(m, fminf(in_a ? inf : ga, in_b || hit_a ? inf : gb));
        node = hit_b ? lb : in_a ? la : in_b ? lb : top;
        const bool push = in_a && in_b, pop = !in_a && !in_b;
        top = push ? lb : pop ? below : top;
        sp += push ? 1 : pop ? -1 : 0;
    } while (node >= 0 && --budget > 0 && sp < kStack);
    if (node >= 0) {
        atomicOr(err, ERR_STACK);
        m = 0.0f;
        return -1;
    }
    if (node == kEmpty) return -1;
    m = fminf(m, hit_a ? box_inner(p, a.a, a.b) : box_inner(p, b.a, b.b));
    return ~node;
}

// The whole first-hit query of one body (root box, single leaf, walk) with its margin.  A NaN
// is in no box, but its answer holds for no other point: margin 0.
__device__ __forceinline__ int query_margin(const BvhRoot* rt, f3 p, int* err, float& m) {
    const f4x2 box = ld8(&rt->top_lo);
    const float4 lo = box.a, hi = box.b;
    if (!in_box(p, lo, hi)) {  // also a NaN
        m = isnan(p.x) || isnan(p.y) || isnan(p.z) ? 0.0f : fminf(m, box_gap(p, lo, hi));
        return -1;
    }
    const int nl = rt->n_leaves;
    if (nl == 1) {
        m = fminf(m, box_inner(p, lo, hi));
        return 0;
    }
    return first_hit(rt->nodes, rt->root, nl, p, err, m);
}

// Force of one spring on the vertex at x moving with velocity vel (verlet.cu:64-84):
//   c = -k (|d| - L0) + kd (dv.d) / |d|,  force = c * normalize(d),  d = x - x_j + FLT_EPSILON
// t0/t1 is the neighbour's record: position and velocity (p2 - p2_old) / dt, stored
// once per step by the neighbour's own thread with the same IEEE division; nk = -k.
// With drec the neighbour's record holds D = p2 - p2_old; its velocity is D / dt.
__device__ __forceinline__ f3 spring_force(f3 x, f3 vel, float4 t0, float4 t1, float nk, float rest, float kd, f3 eps3,
                                           bool drec, float dt) {
    const f3 dP = add(sub(x, mk3(t0.x, t0.y, t0.z)), eps3);
    const float dist = __fsqrt_rn(dot(dP, dP));
    f3 v2 = mk3(t0.w, t1.x, t1.y);
    if (drec) v2 = divs(v2, dt);
    const f3 dV = sub(vel, v2);
    const float c = __fadd_rn(__fmul_rn(nk, __fsub_rn(dist, rest)), __fmul_rn(kd, __fdiv_rn(dot(dV, dP), dist)));
    return mul(c, mul(dP, __frcp_rn(dist)));  // normalize(dP) = dP * (1 / |dP|)
}

// Which springs of a row the packed evaluation may not answer for: the least |dP|^2 and
// damping numerator seen.  While every record is tame the upper ends of their ranges hold by
// themselves (tame), so one minimum a pair of springs stands in for a test and a branch each.
struct PairRange {
    float s = 1.0f;
    uint32_t g = 0xffffffffu;
    __device__ __forceinline__ bool exact() const {
        return __float_as_uint(s) >= kExactLo && g >= 2u * kDivLo - 1u;
    }
};

// Two springs of one vertex at once (spring_force on each spring, operation for
// operation): every quantity of theirs is a packed pair, one spring a lane.  The first
// operation of a spring is a subtraction from x, which writes its result into the pair, so
// packing costs no moves.  Every packed operation rounds each lane as the scalar intrinsic
// would, sqrt_rcp_pair returns __fsqrt_rn / __frcp_rn's bits and div_pair __fdiv_rn's within
// their ranges (rg), so each force is bit-identical to the scalar form in fewer instructions
// (sm_100+ f32x2 arithmetic).  Both c and 1 / |dP| are formed negated, which changes no bit
// of their product but a zero's sign in c, and such a zero adds nothing to the sum.
// Against x and y of one spring in a pair, z apart and a range test with a branch per pair:
// 200 steps of a 64 x 64 sheet 1,376 -> 1,326 us, 512 x 512 sheet 114 -> 110 in 4 steps with
// the output stage; batches (bound by the gathers' latency) unchanged.
// FAST: spring damping exactly +0; else ta1 / tb1 are the second halves of the records
// (the neighbours' velocities; such records never carry D) and kd2 the damping.
template <bool FAST>
__device__ __forceinline__ void spring_pair(f3 x, f3 vel, float4 ta, float4 ta1, float4 tb, float4 tb1, fp2 k2,
                                            float rest_a, float rest_b, fp2 kd2, fp2 eps2, fp2& fx, fp2& fy, fp2& fz,
                                            PairRange& rg) {
    const fp2 dx = add2(pk2(__fsub_rn(x.x, ta.x), __fsub_rn(x.x, tb.x)), eps2);
    const fp2 dy = add2(pk2(__fsub_rn(x.y, ta.y), __fsub_rn(x.y, tb.y)), eps2);
    const fp2 dz = add2(pk2(__fsub_rn(x.z, ta.z), __fsub_rn(x.z, tb.z)), eps2);
    const fp2 s = add_lanes(add_lanes(mul2(dx, dx), mul2(dy, dy)), mul2(dz, dz));  // dot(dP, dP)
    rg.s = fminf(fminf(rg.s, lo2(s)), hi2(s));
    fp2 dist, ninv;
    sqrt_rcp_pair(s, dist, ninv);
    fp2 nc = mul2(k2, pk2(__fsub_rn(lo2(dist), rest_a), __fsub_rn(hi2(dist), rest_b)));  // k (|dP| - L0)
    if (!FAST) {
        const fp2 gx = mul2(pk2(__fsub_rn(vel.x, ta.w), __fsub_rn(vel.x, tb.w)), dx);
        const fp2 gy = mul2(pk2(__fsub_rn(vel.y, ta1.x), __fsub_rn(vel.y, tb1.x)), dy);
        const fp2 gz = mul2(pk2(__fsub_rn(vel.z, ta1.y), __fsub_rn(vel.z, tb1.y)), dz);
        const fp2 g = add_lanes(add_lanes(gx, gy), gz);  // dot(dV, dP)
        rg.g = min(min(rg.g, div_order(lo2(g))), div_order(hi2(g)));
        nc = add_lanes(nc, mul2(kd2, div_pair(g, dist, ninv)));
    }
    fx = mul2(nc, mul2(dx, ninv));
    fy = mul2(nc, mul2(dy, ninv));
    fz = mul2(nc, mul2(dz, ninv));
}

// Contact data a vertex will read after its spring sum (its cached leaf, its stored
// normal), prefetched when the vertex starts: 0 = not prefetched, 1 = into L1, 2 = L2.
// Those reads otherwise start a dependent DRAM round trip at the end of every warp
// with a contact in it; prefetched into L2 the step kernel takes 0.272 ms against
// 0.278 over the 256-garment draped batch (into L1: the same).
constexpr int kPrefetchContact = 2;
__device__ __forceinline__ void prefetch_contact(const void* p) {
    if (kPrefetchContact == 1) asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
    if (kPrefetchContact == 2) asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// Vertex records (about half the neighbour reads hit L1: rows of a grid share most
// neighbours).
struct GlobalRecords {  // by record index (rec_at)
    const float4* p;
    __device__ __forceinline__ float4 r0(uint32_t r) const { return p[r]; }
    __device__ __forceinline__ float4 r1(uint32_t r) const { return p[r + 32u]; }
};
// a record read anew (not merged with an earlier read of it)
__device__ __forceinline__ f4x2 ld_record(const float4* st, int i) {
    const float4* const p = st + rec_at(i);
    return f4x2{ld4(p), ld4(p + 32)};
}
__device__ __forceinline__ void st_record(float4* st, int i, float4 s0, float4 s1) {
    float4* const p = st + rec_at(i);
    p[0] = s0;
    p[32] = s1;
}

// A row's sliced-ELL entries (entry e at p[32 e]): in global memory, or in the tile's
// block that a TMA bulk copy staged in shared memory.
template <bool SMEM>
struct Entries {
    const uint2* p;
    __device__ __forceinline__ uint2 operator[](int e) const { return SMEM ? p[32 * e] : __ldg(p + 32 * e); }
};

// How a row is summed.  SUM_FAST: spring damping exactly +0, packed pairs; SUM_DAMPED: packed
// pairs with damping; SUM_SCALAR: spring by spring, any record form (the general formula,
// also with zero damping: rows that must be recomputed with the damping term).
enum SumMode { SUM_FAST, SUM_DAMPED, SUM_SCALAR };

// Sum of springs [e, end) of one list of a sliced-ELL row (ep/kp at the row's entry
// 0, entries 32 apart), in CSR order, two at a time (independent chains).
template <SumMode MODE, int UNROLL, bool PERK, class Rec, class Ent>
__device__ __forceinline__ f3 list_sum(const Rec& rec, const Ent& ep, const float* __restrict__ kp, int e,
                                       const int end, const float k, f3 x, f3 vel, float kd, f3 eps3, bool drec,
                                       float dt, PairRange& rg) {
    constexpr bool FAST = MODE == SUM_FAST;
    f3 acc = mk3(0.0f, 0.0f, 0.0f);
    if (MODE != SUM_SCALAR) {  // two springs per packed evaluation; the sum stays in CSR order
        const fp2 eps2 = splat2(eps3.x), k2 = splat2(k), kd2 = FAST ? eps2 : splat2(kd);  // kd2 not read with FAST
        auto pair = [&](int ea_at, int eb_at, fp2& fx, fp2& fy, fp2& fz) {
            const uint2 ea = ep[ea_at], eb = ep[eb_at];
            f4x2 ra, rb;
            if (FAST) {
                ra.a = rec.r0(ea.x);
                rb.a = rec.r0(eb.x);
                ra.b = ra.a;
                rb.b = rb.a;
            } else {
                ra = f4x2{rec.r0(ea.x), rec.r1(ea.x)};
                rb = f4x2{rec.r0(eb.x), rec.r1(eb.x)};
            }
            const fp2 kk = PERK ? pk2(__ldg(kp + 32 * ea_at), __ldg(kp + 32 * eb_at)) : k2;
            spring_pair<FAST>(x, vel, ra.a, ra.b, rb.a, rb.b, kk, __uint_as_float(ea.y), __uint_as_float(eb.y), kd2,
                              eps2, fx, fy, fz, rg);
        };
        fp2 fx, fy, fz;
#pragma unroll UNROLL
        for (; e + 1 < end; e += 2) {
            pair(e, e + 1, fx, fy, fz);
            acc = mk3(__fadd_rn(__fadd_rn(acc.x, lo2(fx)), hi2(fx)), __fadd_rn(__fadd_rn(acc.y, lo2(fy)), hi2(fy)),
                      __fadd_rn(__fadd_rn(acc.z, lo2(fz)), hi2(fz)));
        }
        if (e < end) {  // the last of an odd number, in both lanes
            pair(e, e, fx, fy, fz);
            acc = mk3(__fadd_rn(acc.x, lo2(fx)), __fadd_rn(acc.y, lo2(fy)), __fadd_rn(acc.z, lo2(fz)));
        }
        return acc;
    }
    for (; e < end; ++e) {
        const uint2 ea = ep[e];
        const float nk = PERK ? -__ldg(kp + 32 * e) : -k;
        acc = add(acc, spring_force(x, vel, rec.r0(ea.x), rec.r1(ea.x), nk, __uint_as_float(ea.y), kd, eps3, drec, dt));
    }
    return acc;
}

// F + the spring forces of one vertex, list by list as the reference does
// (force += list sum, verlet.cu:148-149); cnt holds the row's per-list counts.
// UNROLL pairs are in flight: 1 where many warps hide the gathers (more registers would
// cost warps) or the registers are few (damped), 2 beside helper warps.
template <SumMode MODE, int UNROLL, bool PERK, class Rec, class Ent>
__device__ __forceinline__ f3 row_lists(const Rec& rec, const Ent& ep, const float* __restrict__ kp, uint2 cnt, f3 x,
                                        f3 vel, f3 F, const StepParams& P, f3 eps3, PairRange& rg) {
    int e = 0;
#pragma unroll
    for (int l = 0; l < VISG_MAX_LISTS; ++l) {
        if (l < P.n_lists) {
            const int n = (int)(((l < 2 ? cnt.x : cnt.y) >> (16 * (l & 1))) & (l == 3 ? 0x7fffu : 0xffffu));
            F = add(F, list_sum<MODE, UNROLL, PERK>(rec, ep, kp, e, e + n, P.list_k[l], x, vel, P.kd, eps3, P.drec != 0,
                                                    P.dt, rg));
            e += n;
        }
    }
    return F;
}
template <SumMode MODE, int UNROLL, class Rec, class Ent>
__device__ __forceinline__ f3 row_forces(const Rec& rec, const Ent& ep, const float* __restrict__ kp, uint2 cnt, f3 x,
                                         f3 vel, f3 F, const StepParams& P, bool perk, f3 eps3, PairRange& rg) {
    return perk ? row_lists<MODE, UNROLL, true>(rec, ep, kp, cnt, x, vel, F, P, eps3, rg)
                : row_lists<MODE, UNROLL, false>(rec, ep, kp, cnt, x, vel, F, P, eps3, rg);
}

// |x| < 3e14 and |v| < 1e15 in every component (false for NaN): while every record
// satisfies this, |dP|^2 < 12 (3e14)^2 < 2^100 and |dv.d| < 3 (2e15)^2 for every spring, and
// RN(dv.d / |d|) is finite (|d| within a factor ~2 of max |d_i| unless it underflows to 0).
constexpr float kTameX = 3e14f;
__device__ __forceinline__ bool tame(f3 x, f3 v) {
    const float m = 1e15f;
    return fabsf(x.x) < kTameX && fabsf(x.y) < kTameX && fabsf(x.z) < kTameX && fabsf(v.x) < m && fabsf(v.y) < m &&
           fabsf(v.z) < m;
}
// the same for a record that carries D = x - x_old (dmax = 0.5e15 dt, so |D / dt| < 1e15)
__device__ __forceinline__ bool tame_d(f3 x, f3 d, float dmax) {
    return fabsf(x.x) < kTameX && fabsf(x.y) < kTameX && fabsf(x.z) < kTameX && fabsf(d.x) < dmax &&
           fabsf(d.y) < dmax && fabsf(d.z) < dmax;
}

// Helper warps (SV_HELP).  A first-hit walk is 10 to 40 dependent node loads of about 0.2 us
// each, and at the end of a step it follows the spring sum.  Where the SMs have room, a
// CTA has as many warps again: while the main warps sum the springs, helper lane j
// answers the query of vertex j where its last displacement would take it again, if the
// vertex's cached answer is unlikely to last (its margin is below twice that
// displacement).  The answer comes with its own margin, so the main lane takes it over as
// it takes a cached one: it holds if the step ends within the margin of the point that was
// asked about, that is if the step's acceleration moved the vertex by less.  What neither
// covers is queried (or queued) as before, by then with the walk's nodes in the L1.
struct HelperAnswers {
    int* leaf;
    float* margin;     // 0: not asked
    float (*point)[3];
};
__device__ __forceinline__ void pair_arrive(int pair) {
    asm volatile("bar.arrive %0, 64;" ::"r"(pair + 1) : "memory");
}
__device__ __forceinline__ void pair_sync(int pair) { asm volatile("bar.sync %0, 64;" ::"r"(pair + 1) : "memory"); }

// With `settled` (no tree has been rebuilt since the launch before) the walk begins already
// while that launch runs, before the wait: from the records it reads, which nobody writes
// until this launch does, two steps ahead.  Whatever those records are, an answer is only
// taken over within its margin (none if they lead to a NaN).
__device__ __forceinline__ f3 step_ahead(const StepParams& P, const f4x2& rec, float steps, float& reach) {
    f3 d = mk3(rec.a.w, rec.b.x, rec.b.y);  // D, or v
    if (!P.drec) d = mul(d, P.dt);
    // what a step is likely to take off the margin: its displacement, and for a vertex that
    // rests (no displacement) what gravity and the springs move it before it is put back
    const float g = 8.0f * P.dt * P.dt * fmaxf(fabsf(P.gx), fmaxf(fabsf(P.gy), fabsf(P.gz)));
    reach = fmaxf(fabsf(d.x), fmaxf(fabsf(d.y), fabsf(d.z))) + g;
    return add(mk3(rec.a.x, rec.a.y, rec.a.z), mul(steps * P.gamma, d));
}
__device__ __forceinline__ void helper_query(const StepArgs& a, const int4 td, const int j, const HelperAnswers& h) {
    const int i = td.y + j;
    const BvhRoot* const rt = a.roots + (td.x & TILE_GARMENT);
    const bool mine = (td.x & TILE_BODY) && i < td.z && !(__ldg(&a.vcount[i].y) & PIN_BIT);
    int leaf = -1;
    float m = 0.0f, reach;
    f3 p = mk3(0.0f, 0.0f, 0.0f);
    if (mine && a.settled) {
        const f4x2 rec = ld_record(a.state_out, i);
        const f3 q = step_ahead(a.p, rec, 2.0f, reach);
        if (!(rec.b.w > 4.0f * reach)) {
            p = q;
            m = __int_as_float(0x7f800000);  // +inf
            leaf = query_margin(rt, p, a.err, m);
        }
    }
    __syncwarp();
    wait_for_earlier_launches();
    if (mine) {
        const f4x2 rec = ld_record(a.state_in, i);
        const f3 q = step_ahead(a.p, rec, 1.0f, reach);
        if (rec.b.w > 2.0f * reach) {
            m = 0.0f;  // the cached answer will do
        } else {
            if (!(m > disp_bound(q, p) + 0.5f * reach)) {
                p = q;
                m = __int_as_float(0x7f800000);
                leaf = query_margin(rt, p, a.err, m);
            }
            if (leaf >= 0) prefetch_contact(rt->leaves + 2 * leaf);
        }
    }
    h.point[j][0] = p.x;
    h.point[j][1] = p.y;
    h.point[j][2] = p.z;
    h.leaf[j] = leaf;
    h.margin[j] = m;
    __syncwarp();
    pair_arrive(j >> 5);
}

struct NoHook {
    __device__ __forceinline__ void operator()() const {}
};

// One thread's vertex i (`active`: it has one; else ii stands in for loads) of garment
// `garment` (a tile's or slice's flags word), whose row's sliced-ELL entry 0 is sb.
// after_sum() is called by the whole warp once its rows are summed.
// State record of vertex i in buffer b: [x.xyz, v.x] [v.y, v.z, flags, 0] with
// v = (x - x_old) / dt.  x_old is x itself when FLAG_XO_IS_X is set (after a
// contact, a pin or update_vertex) and otherwise the previous step's x, which is
// still in the other buffer: the step reads it there before overwriting it.
template <bool COLL, bool KD0, bool SPLIT, bool SMEM_ENT, bool HELP, class Hook>
__device__ __forceinline__ void vertex_step(const StepArgs& a, const int garment, const int i, const bool active,
                                            const int ii, const uint32_t sb, const uint2* ebase, const uint32_t e0,
                                            const int refv, const int check, const int perk, const bool wild,
                                            const HelperAnswers& help, float& my_disp, uint32_t& my_bad,
                                            const Hook& after_sum) {
    constexpr int kPairs = HELP && KD0 ? 2 : 1;
    const GlobalRecords rec{a.state_in};
    const StepParams& P = a.p;
    const f3 grav = mk3(P.gx, P.gy, P.gz);
    const f3 eps3 = mk3(kFltEpsilon, kFltEpsilon, kFltEpsilon);
    const uint32_t ri = rec_at(ii);
    const float4 s0 = rec.r0(ri);
    const f3 x = mk3(s0.x, s0.y, s0.z);
    const uint2 cnt = __ldg(&a.vcount[ii]);
    const bool pinned = (cnt.y & PIN_BIT) != 0u;
    if (COLL && kPrefetchContact) {
        // the record's flags word: start the loads that a cached
        // contact answer and a stored normal need after the spring sum
        const uint32_t fl0 = __float_as_uint(reinterpret_cast<const float*>(a.state_in + ri + 32)[2]);
        const BvhRoot* const rt = a.roots + (garment & TILE_GARMENT);
        if (fl0 & FLAG_LEAF_CACHED) prefetch_contact(rt->leaves + 2 * (fl0 >> LEAF_SHIFT));
        if (fl0 & FLAG_HAS_NORMAL) prefetch_contact(a.normal + ii);
    }
    f3 xn = x, xon = x, nn = mk3(0.0f, 0.0f, 0.0f);
    bool has_n = false;
    uint32_t flags = 0u;
    float margin = 0.0f;
    const bool moves = active && !pinned;
    f3 F = mk3(0.0f, 0.0f, 0.0f);
    bool redo = wild;
    // gravity and force damping.  With drec and force damping exactly +0 the term v * +0 is a
    // signed zero for every tame v, and g m + (+-0) only differs in the sign of a zero
    // component, which the first list's sum (never -0) erases.
    const bool damped = !P.drec || __float_as_uint(P.damp) != 0u || wild;
    const auto outer_force = [&](f3 vel) {
        const f3 f = mul(grav, P.mass);
        return damped ? add(f, mul(vel, P.damp)) : f;
    };
    if (moves) {
        // The zero-damping sum needs only positions: there the rest of the record
        // (v or D, flags, the query cache's margin) is read after the sum, not held in
        // registers across it.
        const float* kp = perk ? a.sellk + sb : nullptr;
        f3 vel = mk3(0.0f, 0.0f, 0.0f);
        if (!KD0 || damped) {
            const float4 s1 = rec.r1(ri);
            const f3 rv = mk3(s0.w, s1.x, s1.y);  // v, or D = x - x_old with drec
            vel = P.drec ? divs(rv, P.dt) : rv;
        }
        const f3 F0 = outer_force(vel);
        const Entries<SMEM_ENT> ep{ebase + (sb - e0)};
        PairRange rg;
        if (KD0) {
            // Spring damping is +0: the reference adds +0 * RN(dv.d / |d|) to every c.
            // Without it c differs at most in the sign of a zero, which changes no sum
            // (a zero force adds nothing to sums that start at +0, which never become -0),
            // as long as RN(dv.d / |d|) is finite (guaranteed while every record is tame;
            // the wild flag says when one was not) or c is not finite (then F is not
            // finite either: such rows are recomputed with the damping term).
            F = row_forces<SUM_FAST, kPairs>(rec, ep, kp, cnt, x, vel, F0, P, perk != 0, eps3, rg);
        } else {
            F = row_forces<SUM_DAMPED, kPairs>(rec, ep, kp, cnt, x, vel, F0, P, perk != 0, eps3, rg);
        }
        redo = redo || !rg.exact();
    }
    if constexpr (!HELP) after_sum();
    if (moves) {
        // the record again (a second read of a line this thread has just read)
        const f4x2 own = ld_record(a.state_in, ii);
        const float4 r0 = own.a, r1 = own.b;
        const f3 rv = mk3(r0.w, r1.x, r1.y);  // v, or D = x - x_old with drec
        flags = __float_as_uint(r1.z);
        margin = r1.w;
        // what the packed evaluation does not answer for, spring by spring (a staged row may
        // be gone by now: from global memory)
        if (redo || !(isfinite(F.x) && isfinite(F.y) && isfinite(F.z))) {
            const f3 vel = P.drec ? divs(rv, P.dt) : rv;
            const Entries<false> ep{a.sell + sb};
            PairRange rg;
            F = row_forces<SUM_SCALAR, 1>(rec, ep, perk ? a.sellk + sb : nullptr, __ldg(&a.vcount[ii]), x, vel,
                                          outer_force(vel), P, perk != 0, eps3, rg);
        }
        // x - x_old: from the record (drec), else from x_old in the other buffer
        f3 xo = x, d = rv;
        if (!P.drec) {
            if (!(flags & FLAG_XO_IS_X)) xo = xyz(a.state_out[rec_at(ii)]);
            d = sub(x, xo);
        }
        f3 np = mk3(0.0f, 0.0f, 0.0f);
        if (flags & FLAG_HAS_NORMAL) np = xyz(a.normal[ii]);
        F = sub(F, mul(dot(np, F), np));  // inelastic response (verlet.cu:151-152)
        const f3 adt = mul(mul(divs(F, P.mass), P.dt), P.dt);
        if (refv) xn = add(sub(add(x, x), xo), adt);  // never with drec
        else xn = add(add(x, mul(P.gamma, d)), adt);
        xon = x;
    }
    // Query cache.  s1.w holds a margin: while the vertex stays within that L-infinity
    // distance of the point its last first-hit query was answered at, the query's
    // answer is unchanged (first_hit's margin) and is reused: no leaf, or the leaf in
    // the flags word (FLAG_LEAF_CACHED), whose plane test is redone at the new position.
    // The margin shrinks by every displacement since (rounded up); 0 = no cache.
    float skin = 0.0f;
    uint32_t leaf_bits = 0u;  // the cached leaf, in the flags word's place (0: no leaf cached)
    if (COLL) {
        const int g = garment & TILE_GARMENT;
        const bool body = (garment & TILE_BODY) != 0;  // the garment has a body (its tree has leaves)
        bool query = false;
        int leaf = -1;
        if (HELP) {
            __syncwarp();
            pair_sync((int)(threadIdx.x >> 5));
        }
        if (body && active && !pinned) {
            float rem = P.margin ? __fsub_rd(margin, disp_bound(xn, x)) : 0.0f;
            if (rem > 0.0f) {
                if (flags & FLAG_LEAF_CACHED) leaf = (int)(flags >> LEAF_SHIFT);
            } else if (HELP && help.margin[threadIdx.x] > 0.0f) {
                const float* q = help.point[threadIdx.x];
                rem = __fsub_rd(help.margin[threadIdx.x], disp_bound(xn, mk3(q[0], q[1], q[2])));
                leaf = help.leaf[threadIdx.x];
            }
            if (rem > 0.0f) {
                skin = rem;
                if (leaf >= 0 && leaf < kLeafCacheMax) leaf_bits = ((uint32_t)leaf << LEAF_SHIFT) | FLAG_LEAF_CACHED;
                else if (leaf >= 0) skin = 0.0f;  // the leaf does not fit the flags word: not cached
            } else {
                leaf = -1;
                query = true;
            }
        }
        if (SPLIT) {
            // queue the queries (one atomic per warp); k_collide answers them with fully
            // populated warps and stores their margins
            const unsigned m = __ballot_sync(0xffffffffu, query);
            if (m) {
                const int lane = (int)(threadIdx.x & 31u), leader = __ffs(m) - 1;
                uint32_t base = 0;
                if (lane == leader) base = atomicAdd(a.cand_count, (uint32_t)__popc(m));
                base = __shfl_sync(0xffffffffu, base, leader);
                if (query) a.cand[base + __popc(m & ((1u << lane) - 1u))] = make_int2(i, g);
            }
        } else if (__any_sync(0xffffffffu, query) && query) {
            float m = __int_as_float(0x7f800000);  // +inf
            leaf = query_margin(a.roots + g, xn, a.err, m);
            if (P.margin) {
                skin = m;
                if (leaf >= 0 && leaf < kLeafCacheMax) leaf_bits = ((uint32_t)leaf << LEAF_SHIFT) | FLAG_LEAF_CACHED;
            }
        }
        if (leaf >= 0) {  // plane test of the first-hit leaf (primitive.cu:110-125)
            const float4* const leaves = a.roots[g].leaves;
            const f4x2 lf = ld8(leaves + 2 * leaf);
            const float4 L0 = lf.a, L1 = lf.b;
            const f3 n = mk3(L0.w, L1.x, L1.y);
            const float d = dot(sub(xn, mk3(L0.x, L0.y, L0.z)), n);
            if (!(d > 0.0f)) {
                const f3 xp = add(xn, mul(__fmul_rn(1.0f, fabsf(d)), n));
                skin = __fsub_rd(skin, disp_bound(xp, xn));
                xn = xp;
                xon = xn;
                nn = n;
                has_n = true;
            }
        }
    }
    bool untamed = false;
    if (active) {
        const bool xo_is_x = pinned || has_n;
        const f3 dn = sub(xn, xon);
        const f3 vn = P.drec ? dn : divs(dn, P.dt);  // what the record carries
        untamed = P.drec ? !tame_d(xn, dn, P.dmax) : !tame(xn, vn);
        const uint32_t fl = (has_n ? FLAG_HAS_NORMAL : 0u) | (xo_is_x ? FLAG_XO_IS_X : 0u) |
                            (skin > 0.0f ? leaf_bits : 0u);
        st_record(a.state_out, i, make_float4(xn.x, xn.y, xn.z, vn.x),
                  make_float4(vn.y, vn.z, __uint_as_float(fl), skin > 0.0f ? skin : 0.0f));
        if (has_n) a.normal[i] = make_float4(nn.x, nn.y, nn.z, 0.0f);
        if (check) {
            const float dd = fmaxf(fabsf(__fsub_rn(xn.x, x.x)),
                                   fmaxf(fabsf(__fsub_rn(xn.y, x.y)), fabsf(__fsub_rn(xn.z, x.z))));
            const f3 vc = P.drec ? divs(dn, P.dt) : vn;
            if (!isfinite(xn.x) || !isfinite(xn.y) || !isfinite(xn.z) || !isfinite(vc.x) || !isfinite(vc.y) ||
                !isfinite(vc.z))
                ++my_bad;
            else
                my_disp = fmaxf(my_disp, dd);
        }
    }
    if (__any_sync(0xffffffffu, untamed) && (threadIdx.x & 31u) == 0u) atomicOr(a.wild, 1u);
}

// ---- TMA bulk copies into shared memory, completed on an mbarrier ----------------------
constexpr int kBarBytes = 256;                 // an 8-byte mbarrier per warp
constexpr uint64_t kWaitNs = 1000000000ull;    // a stage that has not landed after 1 s is an error

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

// one arrival that also announces `bytes` of transactions, then the copy that completes them
__device__ __forceinline__ void bulk_stage(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
        "l"(src), "r"(bytes), "r"(bar)
        : "memory");
}

__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0u;
}

// bounded wait for the phase of the given parity to complete
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    if (mbar_test(bar, parity)) return true;
    const uint64_t t0 = global_ns();
    while (!mbar_test(bar, parity))
        if (global_ns() - t0 > kWaitNs) return false;
    return true;
}

// whether slice sl is staged: it has entries, and they fit a warp's buffer
__device__ __forceinline__ bool slice_staged(const StepArgs& a, const int4 sl) {
    const uint32_t rows = (uint32_t)sl.w >> 6;
    return rows != 0u && 32u * rows <= (uint32_t)a.slice_cap;
}

// One tile's vertices (a thread each), entries read where ebase points.
template <bool COLL, bool KD0, bool SPLIT, bool SMEM_ENT, bool HELP>
__device__ __forceinline__ void tile_step(const StepArgs& a, const int4 td, const uint2* ebase, const uint32_t e0,
                                          const int refv, const int check, const int perk, const bool wild,
                                          const HelperAnswers& help, float& my_disp, uint32_t& my_bad) {
    const int i = td.y + (int)threadIdx.x;
    const bool active = i < td.z;
    const uint32_t sb =
        active ? __ldg(&a.slice_off[td.w + (int)(threadIdx.x >> 5)]) + (uint32_t)(threadIdx.x & 31u) : e0;
    vertex_step<COLL, KD0, SPLIT, SMEM_ENT, HELP>(a, td.x, i, active, active ? i : td.y, sb, ebase, e0, refv, check,
                                                  perk, wild, help, my_disp, my_bad, NoHook());
}

// The fused step.  With STAGED, persistent warps walk the slices (32 vertices of a garment
// and their contiguous sliced-ELL entries): each has a shared-memory buffer for one slice,
// which a TMA bulk copy fills, so every spring's chain starts with a shared-memory load.
// Once a warp has summed its rows nothing reads the buffer any more (rows that must be
// summed again read global memory), so it starts the copy of its next slice and answers
// the queries, stores the records and loads the next vertices while that lands.  A warp
// waits for no other, and half the shared memory of a ring of two buffers leaves the L1,
// which serves the neighbours' records, the rest: 44 garments (two chains) 68.0 -> 61.8 us a
// step against a ring of two tiles a CTA of 128 (9 CTAs an SM in both).  Slices longer than
// the buffer are read from global memory.  Waits are bounded: one that gives up after kWaitNs sets ERR_TIMEOUT,
// waits (again bounded) for the copy in flight, and the warp exits.
//
// HELP: BLOCK more threads are helper warps (above); one tile per CTA.
// Threads per SM that the registers of the staged kernels allow (CTAs of less than 1,024):
// 56 registers.  44 garments, us a step with as many CTAs as fit: 1,024 threads 68.5, 1,152
// 61.8 (13 registers' worth of values that the springs do not use are spilled), 1,280 67.0,
// 1,536 65.1.  Two pairs of springs in flight (UNROLL) 68, the next slice's records
// prefetched 62.7.
constexpr int kStagedThreads = 1152;
// With helper warps 64 registers, so that launches that overlap find room (72: 20 steps of a
// 131 x 127 mesh 245 us, 64: 233).
template <int BLOCK, bool COLL, bool KD0, bool SPLIT, bool STAGED, bool HELP>
__global__ void __launch_bounds__(HELP ? 2 * BLOCK : BLOCK,
                                  STAGED && BLOCK < 1024 ? kStagedThreads / BLOCK : HELP ? 512 / BLOCK : 0)
    k_step(const StepArgs a, const int refv, const int check, const int perk) {
    extern __shared__ __align__(128) unsigned char dyn_smem[];
    __shared__ int s_leaf[HELP ? BLOCK : 1];
    __shared__ float s_margin[HELP ? BLOCK : 1], s_point[HELP ? BLOCK : 1][3];
    const HelperAnswers help{s_leaf, s_margin, s_point};
    float my_disp = 0.0f;
    uint32_t my_bad = 0;
    if constexpr (HELP) {
        // one tile: its springs do not change, so they are on their way before the wait
        const int4 td = __ldg(&a.tiles[blockIdx.x]);
        const int2 tw = __ldg(&a.twin[blockIdx.x]);
        const uint32_t full = smem_addr(dyn_smem);
        const bool staged = tw.y > 0;
        if (threadIdx.x == 0) {
            mbar_init(full, 1u);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            if (staged) bulk_stage(full + kBarBytes, a.sell + (uint32_t)tw.x, (uint32_t)tw.y * 8u, full);
        }
        __syncthreads();
        if (threadIdx.x >= BLOCK) {
            helper_query(a, td, (int)threadIdx.x - BLOCK, help);
            return;
        }
        wait_for_earlier_launches();
        const bool wild = *reinterpret_cast<const volatile uint32_t*>(a.wild) != 0u;
        const bool landed = __all_sync(0xffffffffu, staged && mbar_wait(full, 0u));
        if (landed) {
            tile_step<COLL, KD0, SPLIT, true, HELP>(a, td, reinterpret_cast<const uint2*>(dyn_smem + kBarBytes),
                                                      (uint32_t)tw.x, refv, check, perk, wild, help, my_disp, my_bad);
        } else {
            if (staged && (threadIdx.x & 31u) == 0u) atomicOr(a.err, ERR_TIMEOUT);
            tile_step<COLL, KD0, SPLIT, false, HELP>(a, td, a.sell, 0u, refv, check, perk, wild, help, my_disp,
                                                       my_bad);
            if (staged && threadIdx.x == 0u) mbar_wait(full, 0u);  // the copy in flight, again bounded
        }
    } else if constexpr (!STAGED) {
        wait_for_earlier_launches();
        const bool wild = *reinterpret_cast<const volatile uint32_t*>(a.wild) != 0u;
        for (int tile = blockIdx.x; tile < a.n_tiles; tile += gridDim.x)
            tile_step<COLL, KD0, SPLIT, false, false>(a, __ldg(&a.tiles[tile]), a.sell, 0u, refv, check, perk, wild,
                                                      help, my_disp, my_bad);
    } else {
        const int warp = (int)(threadIdx.x >> 5), lane = (int)(threadIdx.x & 31u);
        const uint32_t bar = smem_addr(dyn_smem) + 8u * (uint32_t)warp;
        const uint32_t buf = smem_addr(dyn_smem) + kBarBytes + (uint32_t)(warp * a.slice_cap) * 8u;
        const uint2* const entries = reinterpret_cast<const uint2*>(dyn_smem + kBarBytes) + warp * a.slice_cap;
        const int stride = (int)gridDim.x * (BLOCK / 32);
        int s = (int)blockIdx.x * (BLOCK / 32) + warp;
        int4 sl = make_int4(0, 0, 0, 0);
        if (s < a.n_slices) sl = __ldg(&a.slices[s]);
        if (lane == 0) {
            mbar_init(bar, 1u);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            if (slice_staged(a, sl)) bulk_stage(buf, a.sell + (uint32_t)sl.z, ((uint32_t)sl.w >> 6) * 256u, bar);
        }
        __syncwarp();
        wait_for_earlier_launches();  // the springs do not change, so the first are on their way
        const bool wild = *reinterpret_cast<const volatile uint32_t*>(a.wild) != 0u;
        uint32_t parity = 0u;
        for (; s < a.n_slices; s += stride) {
            const bool staged = slice_staged(a, sl);
            const int i = sl.y + lane;
            const bool active = lane < (sl.w & 63);
            int4 next = make_int4(0, 0, 0, 0);
            if (staged) {
                if (!__all_sync(0xffffffffu, mbar_wait(bar, parity))) {
                    if (lane == 0) {
                        atomicOr(a.err, ERR_TIMEOUT);
                        mbar_wait(bar, parity);
                    }
                    return;
                }
                parity ^= 1u;
            }
            const auto fetch_next = [&]() {
                __syncwarp();
                if (s + stride < a.n_slices) next = __ldg(&a.slices[s + stride]);
                if (lane == 0 && slice_staged(a, next)) {
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the rows' loads come first
                    bulk_stage(buf, a.sell + (uint32_t)next.z, ((uint32_t)next.w >> 6) * 256u, bar);
                }
                __syncwarp();
            };
            const uint32_t e0 = (uint32_t)sl.z, sb = e0 + (uint32_t)lane;
            const int ii = active ? i : sl.y;
            if (staged)
                vertex_step<COLL, KD0, SPLIT, true, false>(a, sl.x, i, active, ii, sb, entries, e0, refv, check, perk,
                                                           wild, help, my_disp, my_bad, fetch_next);
            else
                vertex_step<COLL, KD0, SPLIT, false, false>(a, sl.x, i, active, ii, sb, a.sell, 0u, refv, check, perk,
                                                            wild, help, my_disp, my_bad, fetch_next);
            sl = next;
        }
    }
    if (check) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            my_disp = fmaxf(my_disp, __shfl_xor_sync(0xffffffffu, my_disp, o));
            my_bad += __shfl_xor_sync(0xffffffffu, my_bad, o);
        }
        if ((threadIdx.x & 31) == 0) {
            if (my_disp > 0.0f) atomicMax(&a.check[0], __float_as_uint(my_disp));
            if (my_bad) atomicAdd(&a.check[1], my_bad);
        }
    }
}

// Split collision (collision_response_projection, verlet.cu:24-50): the queued
// first-hit queries.  The integrate pass has already written each record as if it
// had no contact (flags without a cache, margin 0); a projected vertex gets
// x' += |dist| n, x_old' = x', v' = 0 and its normal; every answered query stores its
// margin (and leaf) for the query cache.
constexpr int COLLIDE_BLOCK = 256;
__global__ void __launch_bounds__(COLLIDE_BLOCK) k_collide(const StepArgs a) {
    const uint32_t n = *a.cand_count;
    const float dt = a.p.dt;
    for (uint32_t k = blockIdx.x * COLLIDE_BLOCK + threadIdx.x; k < n; k += gridDim.x * COLLIDE_BLOCK) {
        const int2 c = a.cand[k];
        const BvhRoot* const rt = a.roots + c.y;
        const f4x2 rec = ld_record(a.state_out, c.x);
        float4 s0 = rec.a, s1 = rec.b;
        f3 xn = mk3(s0.x, s0.y, s0.z);
        float m = __int_as_float(0x7f800000);  // +inf
        const int leaf = query_margin(rt, xn, a.err, m);
        uint32_t fl = __float_as_uint(s1.z);
        float skin = a.p.margin ? m : 0.0f;
        if (leaf >= 0) {
            if (a.p.margin && leaf < kLeafCacheMax) fl |= ((uint32_t)leaf << LEAF_SHIFT) | FLAG_LEAF_CACHED;
            const f4x2 lf = ld8(rt->leaves + 2 * leaf);
            const float4 L0 = lf.a, L1 = lf.b;
            const f3 nrm = mk3(L0.w, L1.x, L1.y);
            const float d = dot(sub(xn, mk3(L0.x, L0.y, L0.z)), nrm);
            if (!(d > 0.0f)) {
                const f3 xp = add(xn, mul(__fmul_rn(1.0f, fabsf(d)), nrm));
                skin = __fsub_rd(skin, disp_bound(xp, xn));
                xn = xp;
                const f3 vn = divs(sub(xn, xn), dt);
                s0 = make_float4(xn.x, xn.y, xn.z, vn.x);
                s1.x = vn.y;
                s1.y = vn.z;
                fl |= FLAG_HAS_NORMAL | FLAG_XO_IS_X;
                a.normal[c.x] = make_float4(nrm.x, nrm.y, nrm.z, 0.0f);
                if (!tame(xn, vn)) atomicOr(a.wild, 1u);
            }
        }
        if (!(skin > 0.0f)) {
            skin = 0.0f;
            fl &= 7u & ~FLAG_LEAF_CACHED;
        }
        st_record(a.state_out, c.x, s0, make_float4(s1.x, s1.y, __uint_as_float(fl), skin));
    }
}

int g_collide_grid = 0;

// the step kernel instance of a variant
using StepKernel = void (*)(const StepArgs, const int, const int, const int);

template <int BLOCK, bool KD0, bool STAGED, bool HELP>
StepKernel step_kernel(bool coll, bool split) {
    if constexpr (HELP) return k_step<BLOCK, true, KD0, false, STAGED, true>;
    if (coll && split) return k_step<BLOCK, true, KD0, true, STAGED, false>;
    if (coll) return k_step<BLOCK, true, KD0, false, STAGED, false>;
    return k_step<BLOCK, false, KD0, false, STAGED, false>;
}

template <int BLOCK>
StepKernel step_kernel(int variant) {
    const bool coll = (variant & SV_COLLIDE) != 0, split = (variant & SV_SPLIT) != 0, kd0 = (variant & SV_KD0) != 0;
    if (variant & SV_STAGED) return kd0 ? step_kernel<BLOCK, true, true, false>(coll, split)
                                        : step_kernel<BLOCK, false, true, false>(coll, split);
    if constexpr (BLOCK <= kHelpBlockMax)
        if (variant & SV_HELP) return kd0 ? step_kernel<BLOCK, true, false, true>(coll, split)
                                          : step_kernel<BLOCK, false, false, true>(coll, split);
    return kd0 ? step_kernel<BLOCK, true, false, false>(coll, split)
               : step_kernel<BLOCK, false, false, false>(coll, split);
}

// largest dynamic shared memory each kernel instance has been opened up to (per device)
std::mutex g_smem_mu;
std::map<std::pair<int, const void*>, int> g_smem_set;

cudaError_t allow_smem(const void* fn, int bytes) {
    if (bytes <= 48 * 1024) return cudaSuccess;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lk(g_smem_mu);
    int& cur = g_smem_set[{dev, fn}];
    if (cur >= bytes) return cudaSuccess;
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) cur = bytes;
    return e;
}

// events recorded right before and after each step-kernel launch of this thread
// (kernel timing; null = none)
thread_local cudaEvent_t t_before_step = nullptr, t_after_step = nullptr;

template <int BLOCK>
cudaError_t launch_block(const StepArgs& a, int variant, int grid, cudaStream_t s) {
    const bool split = (variant & SV_COLLIDE) && (variant & SV_SPLIT);
    // helper warps need a fused step of one tile per CTA, which they stage as a whole
    const bool help = BLOCK <= kHelpBlockMax && (variant & SV_HELP) && !split && !(variant & SV_STAGED) && grid == a.n_tiles;
    const StepKernel fn = step_kernel<BLOCK>(help ? variant : variant & ~SV_HELP);
    const int smem = help ? kBarBytes + 8 * a.win_cap : step_smem_bytes(variant, BLOCK, a.slice_cap);
    cudaError_t e = allow_smem((const void*)fn, smem);
    if (e != cudaSuccess) return e;
    if (split) {
        e = cudaMemsetAsync(a.cand_count, 0, sizeof(uint32_t), s);
        if (e != cudaSuccess) return e;
    }
    if (t_before_step) cudaEventRecord(t_before_step, s);
    // queued collision keeps stream order: a memset comes before the step, the queue's kernel after it
    const bool overlap = help || ((variant & SV_OVERLAP) && !split);
    e = launch_after(fn, grid, help ? 2 * BLOCK : BLOCK, smem, s, overlap, a, (variant & SV_REFV) ? 1 : 0,
                     (variant & SV_CHECK) ? 1 : 0, (variant & SV_PERK) ? 1 : 0);
    if (e != cudaSuccess) return e;
    if (t_after_step) cudaEventRecord(t_after_step, s);
    if (split) {
        if (g_collide_grid == 0) {
            int dev = 0, sms = 0, occ = 0;
            cudaGetDevice(&dev);
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_collide, COLLIDE_BLOCK, 0);
            // two CTAs per SM walk the queue (grid-stride): threads for the usual queue
            // without idle CTAs competing for slots with the other group's step
            g_collide_grid = sms * (occ >= 2 ? 2 : 1);
        }
        k_collide<<<g_collide_grid, COLLIDE_BLOCK, 0, s>>>(a);
    }
    return cudaGetLastError();
}

template <int BLOCK>
int occupancy_block(int variant, int slice_cap) {
    const StepKernel fn = step_kernel<BLOCK>(variant & ~SV_HELP);
    const int smem = step_smem_bytes(variant, BLOCK, slice_cap);
    if (allow_smem((const void*)fn, smem) != cudaSuccess) return 0;
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, BLOCK, smem) != cudaSuccess) return 0;
    return n;
}

__global__ void k_query(BvhView bv, const float* __restrict__ pts, int n, int* leaf, int* inside, float* dist,
                        float* normal, int* err) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const f3 p = mk3(pts[3 * i], pts[3 * i + 1], pts[3 * i + 2]);
    float m = 0.0f;
    const int lf = bv.root->n_leaves > 0 ? query_margin(bv.root, p, err, m) : -1;
    float d = 0.0f;
    f3 nn = mk3(0.0f, 0.0f, 0.0f);
    int in = 0;
    if (lf >= 0) {
        const float4 L0 = bv.leaves[2 * lf], L1 = bv.leaves[2 * lf + 1];
        nn = mk3(L0.w, L1.x, L1.y);
        d = dot(sub(p, mk3(L0.x, L0.y, L0.z)), nn);
        in = !(d > 0.0f);
    }
    if (leaf) leaf[i] = lf;
    if (inside) inside[i] = in;
    if (dist) dist[i] = d;
    if (normal) {
        normal[3 * i] = nn.x;
        normal[3 * i + 1] = nn.y;
        normal[3 * i + 2] = nn.z;
    }
}

__global__ void k_unpack_positions(const float4* st, int64_t v0, int64_t n, float* out) {
    wait_for_earlier_launches();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 s0 = st[rec_at(v0 + i)];
    out[3 * i] = s0.x;
    out[3 * i + 1] = s0.y;
    out[3 * i + 2] = s0.z;
}

__global__ void k_unpack_state(const float4* __restrict__ st, const float4* __restrict__ other,
                               const float4* __restrict__ nr, int64_t v0, int64_t n, float* x, float* xo, float* nrm) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t r = rec_at(v0 + i);
    const float4 s0 = st[r], s1 = st[r + 32];
    const uint32_t fl = __float_as_uint(s1.z);
    if (x) { x[3 * i] = s0.x; x[3 * i + 1] = s0.y; x[3 * i + 2] = s0.z; }
    if (xo) {
        const float4 o = (fl & FLAG_XO_IS_X) ? s0 : other[r];
        xo[3 * i] = o.x; xo[3 * i + 1] = o.y; xo[3 * i + 2] = o.z;
    }
    if (nrm) {
        const float4 v = (fl & FLAG_HAS_NORMAL) ? nr[v0 + i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        nrm[3 * i] = v.x; nrm[3 * i + 1] = v.y; nrm[3 * i + 2] = v.z;
    }
}

// x == nullptr keeps x, etc.  x_old is written into the other buffer and v is
// recomputed as (x - x_old) / dt; a vertex has a stored normal iff it is non-zero.
__global__ void k_pack_state(float4* st, float4* other, float4* nr, int64_t v0, int64_t n, const float* x,
                             const float* xo, const float* nrm, float dt, int drec, float dmax, uint32_t* wild) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t r = rec_at(v0 + i);
    float4 s0 = st[r], s1 = st[r + 32];
    uint32_t fl = __float_as_uint(s1.z) & (FLAG_HAS_NORMAL | FLAG_XO_IS_X);  // no cached answer
    const f3 x0 = mk3(s0.x, s0.y, s0.z);
    const f3 xo0 = (fl & FLAG_XO_IS_X) ? x0 : xyz(other[r]);
    const f3 xv = x ? mk3(x[3 * i], x[3 * i + 1], x[3 * i + 2]) : x0;
    const f3 xov = xo ? mk3(xo[3 * i], xo[3 * i + 1], xo[3 * i + 2]) : xo0;
    const f3 v = drec ? sub(xv, xov) : divs(sub(xv, xov), dt);  // what the record carries
    if (nrm) {
        const float a = nrm[3 * i], b = nrm[3 * i + 1], c = nrm[3 * i + 2];
        const bool h = a != 0.0f || b != 0.0f || c != 0.0f;
        nr[v0 + i] = make_float4(a, b, c, 0.0f);
        fl = (fl & ~FLAG_HAS_NORMAL) | (h ? FLAG_HAS_NORMAL : 0u);
    }
    fl &= ~FLAG_XO_IS_X;
    other[r] = make_float4(xov.x, xov.y, xov.z, 0.0f);
    st[r] = make_float4(xv.x, xv.y, xv.z, v.x);
    st[r + 32] = make_float4(v.y, v.z, __uint_as_float(fl), 0.0f);
    if (drec ? !tame_d(xv, v, dmax) : !tame(xv, v)) atomicOr(wild, 1u);
}

__global__ void k_check_tame(const float4* __restrict__ st, int64_t n, uint32_t* wild) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t r = rec_at(i);
    const float4 s0 = st[r], s1 = st[r + 32];
    if (!tame(mk3(s0.x, s0.y, s0.z), mk3(s0.w, s1.x, s1.y))) atomicOr(wild, 1u);
}

__global__ void k_clear_margin(float4* st, int64_t v0, int64_t v1) {
    const int64_t i = v0 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < v1) reinterpret_cast<float*>(st + rec_at(i) + 32)[3] = 0.0f;
}

__global__ void k_count_contacts(const float4* __restrict__ st, int64_t n, unsigned long long* count) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool c = i < n && (__float_as_uint(st[rec_at(i) + 32].z) & FLAG_HAS_NORMAL);
    const unsigned m = __ballot_sync(0xffffffffu, c);
    if ((threadIdx.x & 31) == 0 && m) atomicAdd(count, (unsigned long long)__popc(m));
}

// update_vertex (simulation.cu:253-257): x = x_old = p, so v = (p - p) / dt; the
// stored contact normal is kept.  moves: {vertex, p} in page-locked host memory, read from
// there, before the wait for earlier launches: two copies in the stream before it took longer
// than the kernel (dragged 64 x 64 sheet 21.8 -> 14.8 us a frame, six frames
// of 24 garments with their read-back, whose copies shared the engines, 388 -> 300).
// The threads run in no order, so where a vertex may be named twice (`claim`) the moves are
// numbered, each claims its vertex for its number, and only the highest writes: within the
// block where one holds all the moves (`alone`), else in a kernel of their own before.
// Unordered moves and a synchronisation, racing -> claimed: 256 24 -> 24 us, 1,000 25 -> 27,
// 262,144 368 -> 400 (929 with the duplicates found on the host; 1,000 in one block of 1,024
// 33).  Ascending indices, noticed while they are packed, name no vertex twice.
constexpr int SET_BLOCK = 256;
__global__ void k_claim_vertices(const float4* moves, int n, uint32_t* claim, uint32_t number) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t v = k < n ? __float_as_uint(__ldcv(&moves[k].x)) : 0u;
    wait_for_earlier_launches();
    if (k < n) atomicMax(claim + v, number + (uint32_t)k);
}
__global__ void k_set_vertices(float4* st, const float4* moves, int n, float dt, uint32_t* wild, uint32_t* claim,
                               uint32_t number, bool alone) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const float4 m = k < n ? __ldcv(moves + k) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    wait_for_earlier_launches();
    if (claim) {
        uint32_t* const c = claim + __float_as_uint(m.x);
        if (alone) {
            if (k < n) atomicMax(c, number + (uint32_t)k);
            __syncthreads();
        }
        if (k < n && __ldcg(c) != number + (uint32_t)k) return;
    }
    if (k >= n) return;
    const int64_t v = rec_at((int64_t)__float_as_uint(m.x));
    const f3 p = mk3(m.y, m.z, m.w);
    const f3 vel = divs(sub(p, p), dt);
    const uint32_t fl = (__float_as_uint(st[v + 32].z) & FLAG_HAS_NORMAL) | FLAG_XO_IS_X;
    st[v] = make_float4(p.x, p.y, p.z, vel.x);
    st[v + 32] = make_float4(vel.y, vel.z, __uint_as_float(fl), 0.0f);
    if (!tame(p, vel)) atomicOr(wild, 1u);
}

inline unsigned grid_for(int64_t n, int b) { return (unsigned)((n + b - 1) / b); }

}  // namespace

namespace {
// Self-test of the staged copies' bounded wait: thread 0 waits on the phase of an
// mbarrier that nothing arrives on; the wait gives up after kWaitNs and the kernel
// records ERR_TIMEOUT and returns (no copy is in flight).
__global__ void k_selftest_mbar_wait(int* err) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(smem_addr(&bar), 1u);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x == 0 && !mbar_wait(smem_addr(&bar), 0u)) atomicOr(err, ERR_TIMEOUT);
}
}  // namespace

namespace {
// Every float s of [2^-100, 2^100) (the range where the step takes the packed square
// root and reciprocal) through sqrt_rcp_pair, against __fsqrt_rn(s) and
// __frcp_rn(__fsqrt_rn(s)).  The other lane of each pair carries a different float of
// the range (s with its low mantissa bits reversed), checked too.  With each root q, div_pair
// against __fdiv_rn on four numerators in its range [2^-60, 2^52 q): any significand and
// exponent, one just below a power of two, the least, and zero (whose quotient may have
// either sign); so every significand of q meets some 800.  cnt[0] = floats checked, cnt[1] =
// mismatches of the root, cnt[2] = of the reciprocal, cnt[3] = of the quotients.
__device__ __forceinline__ float numerator(uint32_t b, float q, int kind) {
    const uint32_t h = b * 2654435761u, lo = kDivLo >> 23, hi = (__float_as_uint(q) >> 23) + 51u;
    const uint32_t e = lo + (h >> 8) % (hi - lo + 1u), sign = h << 31;
    const uint32_t mantissa = kind == 0 ? (h ^ (b * 40503u)) & 0x7fffffu : 0x7fffffu;
    return kind == 3 ? 0.0f : __uint_as_float(sign | (kind == 2 ? kDivLo : e << 23 | mantissa));
}
__device__ __forceinline__ bool same_quotient(float neg, float g, float q) {  // neg = -g / q
    return g == 0.0f ? neg == 0.0f : __float_as_uint(-neg) == __float_as_uint(__fdiv_rn(g, q));
}
__global__ void k_selftest_exact_math(unsigned long long* cnt) {
    unsigned long long n = 0, bad_q = 0, bad_r = 0, bad_d = 0;
    const uint64_t lo = kExactLo, hi = (uint64_t)kExactLo + kExactSpan;
    for (uint64_t u = lo + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; u < hi;
         u += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t b = (uint32_t)u;
        const uint32_t b2 = (b & 0xffff0000u) | (__brev(b) >> 16);  // same exponent, other mantissa
        const float sa = __uint_as_float(b), sb = __uint_as_float(b2);
        fp2 q, nr;
        sqrt_rcp_pair(pk2(sa, sb), q, nr);
        const float qa = __fsqrt_rn(sa), qb = __fsqrt_rn(sb);
        bad_q += (__float_as_uint(lo2(q)) != __float_as_uint(qa)) + (__float_as_uint(hi2(q)) != __float_as_uint(qb));
        bad_r += (__float_as_uint(-lo2(nr)) != __float_as_uint(__frcp_rn(qa))) +
                 (__float_as_uint(-hi2(nr)) != __float_as_uint(__frcp_rn(qb)));
        n += 2;
#pragma unroll 1
        for (int kind = 0; kind < 4; ++kind) {
            const float ga = numerator(b, qa, kind), gb = numerator(b2, qb, kind);
            const fp2 d = div_pair(pk2(ga, gb), q, nr);
            bad_d += !same_quotient(lo2(d), ga, qa) + !same_quotient(hi2(d), gb, qb);
        }
    }
    atomicAdd(&cnt[0], n);
    if (bad_q) atomicAdd(&cnt[1], bad_q);
    if (bad_r) atomicAdd(&cnt[2], bad_r);
    if (bad_d) atomicAdd(&cnt[3], bad_d);
}
}  // namespace

cudaError_t launch_selftest_exact_math(unsigned long long* cnt, cudaStream_t s) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    k_selftest_exact_math<<<sms * 8, 256, 0, s>>>(cnt);
    return cudaGetLastError();
}

cudaError_t launch_selftest_mbar_wait(int* err, cudaStream_t s) {
    k_selftest_mbar_wait<<<1, 32, 0, s>>>(err);
    return cudaGetLastError();
}

void set_step_timing(cudaEvent_t before, cudaEvent_t after) {
    t_before_step = before;
    t_after_step = after;
}

cudaError_t launch_step(const StepArgs& a, int variant, int block, int grid, cudaStream_t s) {
    if (a.n_tiles == 0) return cudaSuccess;
    if (grid <= 0 || grid > a.n_tiles) grid = a.n_tiles;
    switch (block) {
        case 128: return launch_block<128>(a, variant, grid, s);
        case 256: return launch_block<256>(a, variant, grid, s);
        case 512: return launch_block<512>(a, variant, grid, s);
        case 1024: return launch_block<1024>(a, variant, grid, s);
        default: return cudaErrorInvalidValue;
    }
}

int step_smem_bytes(int variant, int block, int slice_cap) {
    return (variant & SV_STAGED) ? kBarBytes + block / 32 * 8 * slice_cap : 0;
}

int step_max_ctas_per_sm(int variant, int block, int slice_cap) {
    switch (block) {
        case 128: return occupancy_block<128>(variant, slice_cap);
        case 256: return occupancy_block<256>(variant, slice_cap);
        case 512: return occupancy_block<512>(variant, slice_cap);
        case 1024: return occupancy_block<1024>(variant, slice_cap);
        default: return 0;
    }
}

cudaError_t launch_query(BvhView v, const float* pts, int n, int* leaf, int* inside, float* dist, float* normal,
                         int* err, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    k_query<<<grid_for(n, 256), 256, 0, s>>>(v, pts, n, leaf, inside, dist, normal, err);
    return cudaGetLastError();
}

cudaError_t launch_unpack_positions(const float4* state, int64_t v0, int64_t n, float* out, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    return launch_after(k_unpack_positions, (int)grid_for(n, 256), 256, 0, s, true, state, v0, n, out);
}

cudaError_t launch_unpack_state(const float4* state, const float4* other, const float4* normal, int64_t v0, int64_t n,
                                float* x, float* xo, float* nrm, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    k_unpack_state<<<grid_for(n, 256), 256, 0, s>>>(state, other, normal, v0, n, x, xo, nrm);
    return cudaGetLastError();
}

cudaError_t launch_check_tame(const float4* state, int64_t n, uint32_t* wild, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    k_check_tame<<<grid_for(n, 256), 256, 0, s>>>(state, n, wild);
    return cudaGetLastError();
}

cudaError_t launch_clear_margin(float4* state, int64_t v0, int64_t v1, cudaStream_t s) {
    if (v1 <= v0) return cudaSuccess;
    k_clear_margin<<<grid_for(v1 - v0, 256), 256, 0, s>>>(state, v0, v1);
    return cudaGetLastError();
}

cudaError_t launch_count_contacts(const float4* state, int64_t n, unsigned long long* count, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    k_count_contacts<<<grid_for(n, 256), 256, 0, s>>>(state, n, count);
    return cudaGetLastError();
}

cudaError_t launch_set_vertices(float4* state, const float4* moves, int n, float dt, uint32_t* wild, uint32_t* claim,
                                uint32_t number, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    const int grid = (int)grid_for(n, SET_BLOCK);
    if (claim && grid > 1) {
        const cudaError_t e = launch_after(k_claim_vertices, grid, SET_BLOCK, 0, s, true, moves, n, claim, number);
        if (e != cudaSuccess) return e;
    }
    return launch_after(k_set_vertices, grid, SET_BLOCK, 0, s, true, state, moves, n, dt, wild, claim, number, grid == 1);
}

cudaError_t launch_pack_state(float4* state, float4* other, float4* normal, int64_t v0, int64_t n, const float* x,
                              const float* xo,
                              const float* nrm, float dt, int drec, float dmax, uint32_t* wild, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    k_pack_state<<<grid_for(n, 256), 256, 0, s>>>(state, other, normal, v0, n, x, xo, nrm, dt, drec,
                                                 dmax, wild);
    return cudaGetLastError();
}

}  // namespace visg
