// visg_adjoint.cu — reverse-mode derivative of the fused step.
//
// One step (verlet.cu:129-161), for a vertex i that is not pinned:
//   v   = (x - xo)/dt
//   F   = m g + c v + sum_e f_e,  f_e = s_e u_e,  d_e = x_i - x_j + eps, L = |d_e|,
//         u_e = d_e/L, s_e = -k_e (L - L0_e) + kd (v_i - v_j).u_e
//   F*  = F - (n.F) n                       (n = contact normal entering the step, frozen)
//   X*  = x + gamma (x - xo) + F*/m dt^2    (gamma = 1: the reference's 2x - xo + a dt^2)
//   contact (frozen active set, plane normal nu):  X = X* - ((X* - p0).nu) nu,  XO = X
//   no contact:                                    X = X*,                      XO = x
// Pinned: X = XO = x.  Given the adjoints (lX, lXO) of a step's outputs, the step's
// inputs receive
//   l*  = Q (lX + lXO) with Q = I - nu nu^T (contact), or l* = lX and lx += lXO
//   lx += (1 + gamma) l*,  lxo -= gamma l*,  dL/dgamma += l*.(x - xo)
//   G   = P (dt^2/m) l*  with P = I - n n^T    (adjoint of the force on i)
//   lx += (c/dt) G, lxo -= (c/dt) G,  dL/dc += G.v
//   every spring e = (i -> j) with adjoint G_i adds to x_i, xo_i and (negated) x_j, xo_j,
//   and dL/dk_e += -(L - L0) u.G_i,  dL/dkd += (dv.u)(u.G_i).
// FP64 arithmetic is what bounds all of it: a GB300 SM retires a warp's double
// instruction in 16 cycles (measured: one per 64 float ones), so the kernels are laid
// out to keep every SM's FP64 pipe busy and to issue each double operation once:
//   * one thread per directed spring, not per vertex: a sheet of a few thousand
//     vertices has too few warps for 152 SMs, and its longest chain is a row of springs;
//   * a vertex's velocity is divided once (by the thread that produces it), not once per
//     spring that reads it, and not at all where nothing needs it;
//   * a spring's derivative is evaluated once per reverse step (k_adj_entry) and kept for
//     both of its ends, which k_adj_vertex sums through the reverse-entry table.
// Kernel times, before (a thread per vertex, 256 a block: 64 of the 152 SMs for a 128 x 128
// sheet; velocities divided per spring; each derivative twice) and now:
//   128 x 128 sheet, 194,052 entries, undamped: step 82 -> 20.1 us, reverse step 182 -> 27.6
//   57 x 43 mesh, 28,224 entries, damped:       step 81 -> 10.2 us, reverse step 160 -> 12.4
// The FP64 pipe's own time for the sheet's operations (50 a spring in the step, 47 in the
// derivative) is 16 and 15 us.
//
// The differentiated trajectory is computed in FP64 (k_step_f64, the same algorithm
// in double, traversing the body's float LBVH with the double position): stiff
// springs stretch by ~1e-6 of the cloth's size, about the resolution of float
// positions, so gradients with respect to stiffness along a float trajectory carry
// percent-level noise.  The contact set the FP64 forward finds is frozen for the
// reverse sweep.
#include <cuda_runtime.h>
#include <stdint.h>

#include "visg_internal.cuh"

namespace visg {

namespace {

// The reverse sweep runs in double: per-spring contributions of both signs cancel
// over hundreds of steps, and float accumulation loses several digits there.
struct V {
    double x, y, z;
};
__device__ __forceinline__ V ld3(const double* p, int64_t i) { return V{p[3 * i], p[3 * i + 1], p[3 * i + 2]}; }
__device__ __forceinline__ void st3(double* p, int64_t i, V v) {
    p[3 * i] = v.x;
    p[3 * i + 1] = v.y;
    p[3 * i + 2] = v.z;
}
__device__ __forceinline__ V operator+(V a, V b) { return V{a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ V operator-(V a, V b) { return V{a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ V operator*(double s, V a) { return V{s * a.x, s * a.y, s * a.z}; }
__device__ __forceinline__ double dotv(V a, V b) { return a.x * b.x + a.y * b.y + a.z * b.z; }

constexpr double kEps = 1.1920928955078125e-07;

// p as two floats, rounded down and up: for a float bound b, p >= b exactly when
// RD(p) >= b and p <= b exactly when RU(p) <= b, so a box test needs no double compare
struct FloatPair {
    f3 dn, up;
};
__device__ __forceinline__ bool in_box_d(const FloatPair& p, float4 lo, float4 hi) {
    return (p.dn.x >= lo.x && p.up.x <= hi.x) && (p.dn.y >= lo.y && p.up.y <= hi.y) &&
           (p.dn.z >= lo.z && p.up.z <= hi.z);
}

// first-hit traversal (cudaBRT.cu:239-285) of the float tree for a double point
__device__ int first_hit_d(const BvhView& bv, V q, int* err) {
    const FloatPair p{mk3(__double2float_rd(q.x), __double2float_rd(q.y), __double2float_rd(q.z)),
                      mk3(__double2float_ru(q.x), __double2float_ru(q.y), __double2float_ru(q.z))};
    const int nl = bv.root->n_leaves;
    if (nl <= 0 || !in_box_d(p, bv.root->top_lo, bv.root->top_hi)) return -1;
    if (nl == 1) return 0;
    int stack[32];
    int sp = 0, node = bv.root->root, budget = nl;
    while (true) {
        if (--budget < 0) {
            atomicOr(err, ERR_STACK);
            return -1;
        }
        const f4x2 a = ld8_nc(&bv.nodes[node].a_lo), b = ld8_nc(&bv.nodes[node].b_lo);
        const int la = __float_as_int(a.a.w), lb = __float_as_int(b.a.w);
        const bool ol = in_box_d(p, a.a, a.b), orr = in_box_d(p, b.a, b.b);
        if (ol && la < 0) return ~la;
        if (orr && lb < 0) return ~lb;
        const bool tl = ol && la >= 0, tr = orr && lb >= 0;
        if (!tl && !tr) {
            if (sp == 0) return -1;
            node = stack[--sp];
        } else {
            node = tl ? la : lb;
            if (tl && tr) {
                if (sp == 32) {
                    atomicOr(err, ERR_STACK);
                    return -1;
                }
                stack[sp++] = lb;
            }
        }
    }
}

// One step in double, operation by operation the FP64 oracle's arithmetic (the
// reference's expressions evaluated in double with one rounding per operation), so
// the GPU's differentiable trajectory and contact set equal the oracle's bit for bit.
struct R {
    double x, y, z;
};
__device__ __forceinline__ R radd(R a, R b) { return R{__dadd_rn(a.x, b.x), __dadd_rn(a.y, b.y), __dadd_rn(a.z, b.z)}; }
__device__ __forceinline__ R rsub(R a, R b) { return R{__dsub_rn(a.x, b.x), __dsub_rn(a.y, b.y), __dsub_rn(a.z, b.z)}; }
__device__ __forceinline__ R rmul(R a, double s) { return R{__dmul_rn(a.x, s), __dmul_rn(a.y, s), __dmul_rn(a.z, s)}; }
__device__ __forceinline__ R rmul(double s, R a) { return R{__dmul_rn(s, a.x), __dmul_rn(s, a.y), __dmul_rn(s, a.z)}; }
__device__ __forceinline__ R rdiv(R a, double s) { return R{__ddiv_rn(a.x, s), __ddiv_rn(a.y, s), __ddiv_rn(a.z, s)}; }
__device__ __forceinline__ double rdot(R a, R b) {
    return __dadd_rn(__dadd_rn(__dmul_rn(a.x, b.x), __dmul_rn(a.y, b.y)), __dmul_rn(a.z, b.z));
}
__device__ __forceinline__ R rnormalize(R v) { return rmul(v, __ddiv_rn(1.0, __dsqrt_rn(rdot(v, v)))); }
__device__ __forceinline__ R rcross(R a, R b) {
    return R{__dsub_rn(__dmul_rn(a.y, b.z), __dmul_rn(b.y, a.z)), __dsub_rn(__dmul_rn(a.z, b.x), __dmul_rn(b.z, a.x)),
             __dsub_rn(__dmul_rn(a.x, b.y), __dmul_rn(b.x, a.y))};
}
__device__ __forceinline__ R rld(const double* p, int64_t i) { return R{p[3 * i], p[3 * i + 1], p[3 * i + 2]}; }
__device__ __forceinline__ void rst(double* p, int64_t i, R v) {
    p[3 * i] = v.x;
    p[3 * i + 1] = v.y;
    p[3 * i + 2] = v.z;
}
__device__ __forceinline__ R rf4(float4 v) { return R{v.x, v.y, v.z}; }

// (the range test of the float step's `tame`, with room for dt in the velocity: below it
// no product or quotient of the damping term overflows; an integer compare of the
// exponent, so it costs the FP64 pipe nothing)
__device__ __forceinline__ bool tame64(double v) { return (__double2hiint(v) & 0x7fffffff) < 0x54b00000; }  // < ~1e100
__device__ __forceinline__ bool finite64(double v) { return (__double2hiint(v) & 0x7ff00000) != 0x7ff00000; }

// The FP64 step.  A CTA takes `per` (at most F64_VERTS) consecutive vertices, chosen so
// that the CTAs fill the SMs in whole rounds.  Their springs are one contiguous run of
// the merged CSR, taken F64_CHUNK at a time: a thread per spring leaves the spring's
// force in shared memory, then a thread per vertex component adds its row's forces in
// CSR order (one rounding per addition, as the reference sums) and finishes the
// integration of that component; a thread per vertex does the contact query.
// KD: the springs are damped; velocities come from the array the previous step wrote.
// Without KD the damping term is +0 * RN(dv.d / |d|): it changes no sum while every
// component is tame (the argument of the float step), so it is left out until the `wild`
// word says one was not.
constexpr int F64_THREADS = 128;
constexpr int F64_VERTS = 32;
constexpr int F64_CHUNK = 3 * F64_THREADS;
template <bool KD>
__global__ void __launch_bounds__(F64_THREADS) k_step_f64(const Step64Args a, const int per) {
    __shared__ double s_f[3 * F64_CHUNK];
    __shared__ uint32_t s_list[F64_CHUNK];
    __shared__ uint32_t s_row[F64_VERTS + 1];
    __shared__ double s_x[3 * F64_VERTS], s_xo[3 * F64_VERTS], s_v[3 * F64_VERTS], s_F[3 * F64_VERTS];
    __shared__ double s_n[3 * F64_VERTS];
    const StepParams& P = a.p;
    const int tid = (int)threadIdx.x;
    const int64_t i0 = (int64_t)blockIdx.x * per;
    const int nv = (int)min((int64_t)per, (int64_t)a.n - i0);
    // one read for the whole CTA: another CTA of this launch may set the word meanwhile
    const bool wild = __syncthreads_or(tid == 0 && *reinterpret_cast<const volatile uint32_t*>(a.wild) != 0u) != 0;
    const bool need_v = KD || wild || __float_as_uint(P.damp) != 0u;
    const double dt = P.dt, mass = P.mass, kd = P.kd, eps = kEps;
    if (tid <= nv) s_row[tid] = a.rowp[i0 + tid];  // with the pin bit
    const bool comp = tid < 3 * nv;                // this thread's vertex component
    const int vi = tid / 3, c = tid - 3 * vi;
    if (comp) {
        const double x = a.x[3 * i0 + tid], xo = a.xo[3 * i0 + tid];
        s_x[tid] = x;
        s_xo[tid] = xo;
        s_n[tid] = a.n_in[3 * i0 + tid];
        if (need_v) s_v[tid] = KD ? a.v[3 * i0 + tid] : __ddiv_rn(__dsub_rn(x, xo), dt);
    }
    __syncthreads();
    double force = 0.0, acc = 0.0;
    int list = 0;
    uint32_t le = 0, lend = 0;
    bool pinned = false;
    if (comp) {
        pinned = (s_row[vi] & PIN_BIT) != 0u;
        le = s_row[vi] & ROW_MASK;
        lend = s_row[vi + 1] & ROW_MASK;
        force = __dmul_rn((double)(c == 0 ? P.gx : c == 1 ? P.gy : P.gz), mass);
        // force damping of exactly +0 adds a signed zero, which the first list's sum erases
        if (need_v) force = __dadd_rn(force, __dmul_rn(s_v[tid], (double)P.damp));
    }
    const uint32_t e0 = s_row[0] & ROW_MASK, e1 = s_row[nv] & ROW_MASK;
    for (uint32_t cb = e0; cb < e1; cb += F64_CHUNK) {
        const uint32_t ce = min(cb + (uint32_t)F64_CHUNK, e1);
        for (uint32_t e = cb + tid; e < ce; e += F64_THREADS) {
            const int li = (int)((int64_t)__ldg(a.src + e) - i0);
            const uint32_t w = __ldg(&a.ent[e].x);
            s_list[e - cb] = w >> LIST_SHIFT;
            if (s_row[li] & PIN_BIT) continue;
            const uint32_t j = w & END_MASK;
            const double ks = a.k64 ? __ldg(a.k64 + e) : a.list_k[w >> LIST_SHIFT];
            const R p2 = rld(a.x, j);
            const R dP = radd(rsub(R{s_x[3 * li], s_x[3 * li + 1], s_x[3 * li + 2]}, p2), R{eps, eps, eps});
            const double dist = __dsqrt_rn(rdot(dP, dP));
            double s = __dmul_rn(-ks, __dsub_rn(dist, __ldg(a.rest64 + e)));
            if (KD || wild) {
                const R v2 = KD ? rld(a.v, j) : rdiv(rsub(p2, rld(a.xo, j)), dt);
                const R dV = rsub(R{s_v[3 * li], s_v[3 * li + 1], s_v[3 * li + 2]}, v2);
                s = __dadd_rn(s, __dmul_rn(kd, __ddiv_rn(rdot(dV, dP), dist)));
            }
            rst(s_f, e - cb, rmul(s, rmul(dP, __drcp_rn(dist))));
        }
        __syncthreads();
        if (comp && !pinned) {
            const uint32_t re = min(lend, ce);
            for (; le < re; ++le) {
                const int f = (int)s_list[le - cb];
                while (list < f) {
                    force = __dadd_rn(force, acc);
                    acc = 0.0;
                    ++list;
                }
                acc = __dadd_rn(acc, s_f[3 * (le - cb) + c]);
            }
        }
        if (ce < e1) __syncthreads();
    }
    if (comp) {
        while (list < P.n_lists) {
            force = __dadd_rn(force, acc);
            acc = 0.0;
            ++list;
        }
        s_F[tid] = force;
    }
    __syncthreads();
    double pos = 0.0, pos0 = 0.0;
    if (comp) {
        pos0 = s_x[tid];
        pos = pos0;
        if (!pinned) {
            const R F{s_F[3 * vi], s_F[3 * vi + 1], s_F[3 * vi + 2]};
            const R cf{s_n[3 * vi], s_n[3 * vi + 1], s_n[3 * vi + 2]};
            // a zero normal leaves a finite force as it is
            if (cf.x != 0.0 || cf.y != 0.0 || cf.z != 0.0 || !finite64(F.x) || !finite64(F.y) || !finite64(F.z))
                force = __dsub_rn(force, __dmul_rn(rdot(cf, F), s_n[tid]));
            const double adt = __dmul_rn(__dmul_rn(__ddiv_rn(force, mass), dt), dt);
            pos = a.refv ? __dadd_rn(__dsub_rn(__dadd_rn(pos0, pos0), s_xo[tid]), adt)
                         : __dadd_rn(__dadd_rn(pos0, __dmul_rn((double)P.gamma, __dsub_rn(pos0, s_xo[tid]))), adt);
        }
    }
    // s_xo, s_n: from here on the step's x_old and contact normal
    __syncthreads();
    if (comp) {
        s_F[tid] = pos;
        s_xo[tid] = pos0;
        s_n[tid] = 0.0;
    }
    if (a.collide && a.bodies[0].root != nullptr) {
        __syncthreads();
        bool hit = false;
        if (tid < nv && !(s_row[tid] & PIN_BIT)) {
            R p{s_F[3 * tid], s_F[3 * tid + 1], s_F[3 * tid + 2]};
            const int leaf = first_hit_d(a.bodies[0], V{p.x, p.y, p.z}, a.err);
            if (leaf >= 0) {
                const int t = __float_as_int(a.bodies[0].leaves[2 * leaf + 1].z);
                const R v0 = rf4(a.body_verts[a.body_tris[3 * t]]), v1 = rf4(a.body_verts[a.body_tris[3 * t + 1]]),
                        v2 = rf4(a.body_verts[a.body_tris[3 * t + 2]]);
                const R normal = rnormalize(rcross(rsub(v1, v0), rsub(v2, v0)));
                double dist = rdot(rsub(p, v0), normal);
                if (!(dist > 0.0)) {
                    dist = __dmul_rn(1.0, fabs(dist));
                    p = radd(p, rmul(dist, normal));
                    rst(s_F, tid, p);
                    rst(s_xo, tid, p);
                    rst(s_n, tid, normal);
                    hit = normal.x != 0.0 || normal.y != 0.0 || normal.z != 0.0;
                }
            }
        }
        if (a.contacts && tid < 32) {  // vertices projected in this step (all in the first warp)
            const unsigned m = __ballot_sync(0xffffffffu, hit);
            if (m && tid == 0) atomicAdd(a.contacts, (unsigned)__popc(m));
        }
        __syncthreads();
    }
    if (comp) {
        const double xn = s_F[tid], xon = s_xo[tid];
        a.xn[3 * i0 + tid] = xn;
        a.xon[3 * i0 + tid] = xon;
        a.n_out[3 * i0 + tid] = s_n[tid];
        if (KD) a.vn[3 * i0 + tid] = __ddiv_rn(__dsub_rn(xn, xon), dt);
        if (!tame64(xn) || !tame64(xon)) atomicOr(a.wild, 1u);
    }
}

// the velocities (and the wild word) of a state that the step did not write
__global__ void k_vel_f64(const double* __restrict__ x, const double* __restrict__ xo, double* __restrict__ v, float dt,
                          uint32_t* wild, int64_t n3) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n3) return;
    if (v) v[k] = __ddiv_rn(__dsub_rn(x[k], xo[k]), (double)dt);
    if (!tame64(x[k]) || !tame64(xo[k])) atomicOr(wild, 1u);
}

__global__ void k_widen(const float* __restrict__ src, double* __restrict__ dst, int64_t n) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) dst[k] = (double)src[k];
}

__global__ void k_narrow(const double* __restrict__ src, float* __restrict__ dst, int64_t n) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) dst[k] = (float)src[k];
}

// rest lengths and stiffnesses as doubles (a conversion takes a slot of the FP64 pipe, so
// the steps do not repeat it)
__global__ void k_entries_f64(const uint2* __restrict__ ent, const float* __restrict__ kent, double* __restrict__ rest,
                              double* __restrict__ k64, int64_t n) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n) return;
    rest[e] = (double)__uint_as_float(ent[e].y);
    if (k64) k64[e] = (double)kent[e];
}

// the gradient per entry in the caller's order, as floats; *bad counts those that are not finite
__global__ void k_adj_result(const double* __restrict__ dk, const uint32_t* __restrict__ pos, float* __restrict__ out,
                             unsigned* bad, int64_t n) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const float v = k < n ? (float)dk[k] : 0.0f;
    if (k < n) out[pos[k]] = v;
    const unsigned m = __ballot_sync(0xffffffffu, !isfinite(v));
    if (m && (threadIdx.x & 31u) == 0u) atomicAdd(bad, (unsigned)__popc(m));
}

// Per spring e = (i -> j) of the step: its contributions to x_i and x_old_i (negated: to
// x_j, x_old_j), dL/dk_e and dL/dkd.  One thread per spring: ~55 double operations each
// fill the FP64 pipes whatever the sheet's size.  With u = d / L, r = 1 / L:
//   a = s / L,  gx = a G + (uG (-k - a)) u,  dL/dk = -(L - L0) uG,  dL/dkd = (dv.u) uG
// and with damping  gx += (kd uG / L) (dv - (dv.u) u) + h,  gxo = -h,  h = (kd uG / dt) u.
// FULL: the springs are damped, or some state was not tame (then the damping terms' NaNs
// must come out as written); two bodies, so that the undamped one issues none of the rest.
constexpr int ADJ_THREADS = 128;
__device__ __forceinline__ bool adj_full(const AdjArgs& a) {
    return a.gxo != nullptr && (__float_as_uint(a.p.kd) != 0u || *a.wild != 0u);
}
template <bool FULL>
__device__ __forceinline__ void adj_entry(const AdjArgs& a, const uint32_t e) {
    const uint32_t i = __ldg(a.src + e), r = __ldg(a.rev + e);
    V gx{0, 0, 0}, gxo{0, 0, 0};
    if (!(__ldg(a.rowp + i) & PIN_BIT)) {  // a pinned vertex's springs have no adjoint
        const uint32_t w = __ldg(&a.ent[e].x), j = w & END_MASK;
        const double k = a.k64 ? __ldg(a.k64 + e) : a.list_k[w >> LIST_SHIFT];
        const V d = (ld3(a.x, i) - ld3(a.x, j)) + V{kEps, kEps, kEps};
        const V dv = ld3(a.v, i) - ld3(a.v, j);
        const V G = ld3(a.G, i);
        const double dd = dotv(d, d);
        const double rl = rsqrt(dd);
        double L = dd * rl;
        L = fma(fma(-L, L, dd), 0.5 * rl, L);  // the square root's last bits
        const V u = rl * d;
        const double dvu = dotv(dv, u), uG = dotv(u, G);
        const double ext = L - __ldg(a.rest64 + e);
        double s = -k * ext;
        if (FULL) s = fma(a.kd, dvu, s);
        const double al = s * rl, be = uG * (-k - al);
        gx = V{fma(al, G.x, be * u.x), fma(al, G.y, be * u.y), fma(al, G.z, be * u.z)};
        if (FULL) {
            const double kuG = a.kd * uG, kh = kuG * a.inv_dt, kr = kuG * rl;
            gxo = V{-kh * u.x, -kh * u.y, -kh * u.z};
            gx = V{fma(kr, fma(-dvu, u.x, dv.x), gx.x) - gxo.x, fma(kr, fma(-dvu, u.y, dv.y), gx.y) - gxo.y,
                   fma(kr, fma(-dvu, u.z, dv.z), gx.z) - gxo.z};
        }
        a.dk[e] = fma(-ext, uG, a.dk[e]);
        a.dkd[e] = fma(dvu, uG, a.dkd[e]);
    }
    st3(a.gx, 2 * (int64_t)e, gx);
    st3(a.gx, 2 * (int64_t)r + 1, V{-gx.x, -gx.y, -gx.z});
    if (FULL) {
        st3(a.gxo, 2 * (int64_t)e, gxo);
        st3(a.gxo, 2 * (int64_t)r + 1, V{-gxo.x, -gxo.y, -gxo.z});
    }
}
__global__ void __launch_bounds__(ADJ_THREADS) k_adj_entry(const AdjArgs a) {
    const int64_t e = (int64_t)blockIdx.x * ADJ_THREADS + threadIdx.x;
    if (e >= a.E) return;
    if (adj_full(a))
        adj_entry<true>(a, (uint32_t)e);
    else
        adj_entry<false>(a, (uint32_t)e);
}

// Per vertex: the adjoint of the step's outputs is complete once the springs of the step
// after it have been added (each entry's own contribution, and the negated one of its
// reverse entry, which that entry has left beside it); from it follow the adjoint of the
// vertex's own terms of the step's inputs and of its force, G.  A double addition has a
// long latency and a sheet has few vertices, so a row is summed by ADJ_PARTS threads per
// component; a thread per component then finishes, packed into the block's first warps.
constexpr int ADJ_VERTS = 16;
constexpr int ADJ_PARTS = 4;
__global__ void __launch_bounds__(3 * ADJ_VERTS * ADJ_PARTS) k_adj_vertex(const AdjArgs a) {
    __shared__ double s_lx[3 * ADJ_VERTS], s_lxo[3 * ADJ_VERTS];
    const StepParams& P = a.p;
    const int tid = (int)threadIdx.x;
    const bool full = adj_full(a);
    const int64_t i0 = (int64_t)blockIdx.x * ADJ_VERTS;
    {
        const int q = tid % ADJ_PARTS, t = tid / ADJ_PARTS, vi = t / 3, c = t - 3 * vi;
        const int64_t i = i0 + vi;
        double lX = 0.0, lXO = 0.0;
        if (i < a.n) {
            if (q == 0) {
                lX = a.lx[3 * i + c];
                lXO = a.lxo[3 * i + c];
            }
            if (a.gather) {
                const uint32_t re = __ldg(a.rowp + i + 1) & ROW_MASK;
#pragma unroll 4
                for (uint32_t e = (__ldg(a.rowp + i) & ROW_MASK) + q; e < re; e += ADJ_PARTS) {
                    const double* g = a.gx + 6 * (int64_t)e + c;
                    lX += g[0] + g[3];
                    if (full) {
                        const double* go = a.gxo + 6 * (int64_t)e + c;
                        lXO += go[0] + go[3];
                    }
                }
            }
        }
#pragma unroll
        for (int o = ADJ_PARTS / 2; o > 0; o >>= 1) {
            lX += __shfl_xor_sync(0xffffffffu, lX, o);
            if (full) lXO += __shfl_xor_sync(0xffffffffu, lXO, o);
        }
        if (q == 0) {
            s_lx[t] = lX;
            s_lxo[t] = lXO;
        }
    }
    __syncthreads();
    const int vi = tid / 3, c = tid - 3 * vi;
    const int64_t i = i0 + vi;
    if (tid >= 3 * ADJ_VERTS || i >= a.n) return;
    const double lX = s_lx[tid], lXO = s_lxo[tid], gam = P.gamma;
    const double d = a.x[3 * i + c] - a.xo[3 * i + c], v = a.inv_dt * d;
    double lx = 0.0, lxo = 0.0, G = 0.0;
    if (__ldg(a.rowp + i) & PIN_BIT) {
        lx = lX + lXO;
    } else {
        const V nu = ld3(a.n_out, i), np = ld3(a.n_in, i);
        double ls = lX;
        V l{s_lx[3 * vi], s_lx[3 * vi + 1], s_lx[3 * vi + 2]};
        if (nu.x != 0.0 || nu.y != 0.0 || nu.z != 0.0) {
            const V s = l + V{s_lxo[3 * vi], s_lxo[3 * vi + 1], s_lxo[3 * vi + 2]};
            l = s - dotv(nu, s) * nu;
            ls = c == 0 ? l.x : c == 1 ? l.y : l.z;
        } else {
            lx = lXO;
        }
        G = a.dt2_mass * ls;
        if (np.x != 0.0 || np.y != 0.0 || np.z != 0.0)
            G -= (a.dt2_mass * dotv(np, l)) * (c == 0 ? np.x : c == 1 ? np.y : np.z);
        const double gl = gam * ls, q = a.damp_dt * G;
        lx += ls + gl + q;
        lxo = -gl - q;
        a.dgc[2 * (3 * i + c)] = fma(ls, d, a.dgc[2 * (3 * i + c)]);
        a.dgc[2 * (3 * i + c) + 1] = fma(G, v, a.dgc[2 * (3 * i + c) + 1]);
    }
    a.lx[3 * i + c] = lx;
    a.lxo[3 * i + c] = lxo;
    a.G[3 * i + c] = G;
    a.v[3 * i + c] = v;
}

// dscalar[3] += the sums of the per-component and per-entry parts
__global__ void __launch_bounds__(256) k_adj_scalars(const double* __restrict__ dgc, int64_t n3,
                                                     const double* __restrict__ dkd, int64_t E, double* dscalar) {
    double s[3] = {0.0, 0.0, 0.0};
    const int64_t k0 = (int64_t)blockIdx.x * 256 + threadIdx.x, step = (int64_t)gridDim.x * 256;
    for (int64_t k = k0; k < n3; k += step) {
        s[0] += dgc[2 * k];
        s[1] += dgc[2 * k + 1];
    }
    for (int64_t k = k0; k < E; k += step) s[2] += dkd[k];
    for (int j = 0; j < 3; ++j) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s[j] += __shfl_xor_sync(0xffffffffu, s[j], o);
        if ((threadIdx.x & 31) == 0 && s[j] != 0.0) atomicAdd(&dscalar[j], s[j]);
    }
}

}  // namespace

cudaError_t launch_step_f64(const Step64Args& a, cudaStream_t s) {
    if (a.n <= 0) return cudaSuccess;
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    // vertices per CTA: the fewest rounds of one CTA per SM that F64_VERTS allows, evenly cut
    const int rounds = (a.n + sms * F64_VERTS - 1) / (sms * F64_VERTS);
    const int per = (a.n + sms * rounds - 1) / (sms * rounds);
    const int grid = (a.n + per - 1) / per;
    if (a.v)
        k_step_f64<true><<<grid, F64_THREADS, 0, s>>>(a, per);
    else
        k_step_f64<false><<<grid, F64_THREADS, 0, s>>>(a, per);
    return cudaGetLastError();
}

cudaError_t launch_vel_f64(const double* x, const double* xo, double* v, float dt, uint32_t* wild, int64_t n3,
                           cudaStream_t s) {
    if (n3 <= 0) return cudaSuccess;
    k_vel_f64<<<(unsigned)((n3 + 255) / 256), 256, 0, s>>>(x, xo, v, dt, wild, n3);
    return cudaGetLastError();
}

cudaError_t launch_widen(const float* src, double* dst, int64_t n, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    k_widen<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(src, dst, n);
    return cudaGetLastError();
}

cudaError_t launch_narrow(const double* src, float* dst, int64_t n, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    k_narrow<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(src, dst, n);
    return cudaGetLastError();
}

cudaError_t launch_entries_f64(const uint2* ent, const float* kent, double* rest, double* k64, int64_t n,
                               cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    k_entries_f64<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(ent, kent, rest, k64, n);
    return cudaGetLastError();
}

cudaError_t launch_adj_scalars(const double* dgc, int64_t n3, const double* dkd, int64_t E, double* dscalar,
                               cudaStream_t s) {
    k_adj_scalars<<<64, 256, 0, s>>>(dgc, n3, dkd, E, dscalar);
    return cudaGetLastError();
}

cudaError_t launch_adj_result(const double* dk, const uint32_t* pos, float* out, unsigned* bad, int64_t n,
                              cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    k_adj_result<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(dk, pos, out, bad, n);
    return cudaGetLastError();
}

cudaError_t launch_adjoint_step(const AdjArgs& a, cudaStream_t s) {
    if (a.n <= 0) return cudaSuccess;
    k_adj_vertex<<<(unsigned)((a.n + ADJ_VERTS - 1) / ADJ_VERTS), 3 * ADJ_VERTS * ADJ_PARTS, 0, s>>>(a);
    if (a.E > 0) k_adj_entry<<<(unsigned)((a.E + ADJ_THREADS - 1) / ADJ_THREADS), ADJ_THREADS, 0, s>>>(a);
    return cudaGetLastError();
}

}  // namespace visg
