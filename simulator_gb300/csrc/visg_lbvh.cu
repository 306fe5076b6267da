// visg_lbvh.cu — per-step body LBVH build on the device, in one launch.
//
// Reference (BVHAccel, src/bvh/bvh.cu:154-297; cudaBRT.cu:9-206) builds once per
// body with a device->host->device round trip: expanded boxes and Morton codes on
// the GPU, std::sort + duplicate removal on the CPU, then Karras internal nodes and
// an atomic-counter refit on the GPU.  Here the whole build is one cooperative
// launch of k_rebuild, so it can run every step: persistent CTAs, all resident at
// once, walk its phases, and a grid barrier (every CTA arrives on a counter, then
// waits for the others, bounded) separates phases that read what others wrote:
//   verts   vertex_extend (Mesh.cpp:101-117) v += thickness * n, stored as float4
//           (the same launch voids the query-cache margins of the body's cloth); a small
//           body's triangles gather the caller's vertices themselves and do not wait for it
//   boxes   expanded triangle boxes (primitive.cu:79-91) and leaf records, three
//           corners gathered as aligned float4; per CTA the union of its boxes
//           with the identity box
//   codes   the Morton frame (identity box U every box: each CTA reduces the CTA
//           unions itself); the Morton code of each box centroid in the frame
//           (bvh.cu:20-41,71-79; bbox.h:97-127); codes that differ from the last
//           build's are listed
//   sort    the order by (code, triangle), one of three ways.  The last build's sorted list
//           is at hand and at most CHG_CAP codes changed (a body that moves
//           rigidly flips a few codes at cell edges): it is merged; the unchanged
//           entries keep their order, every CTA sorts the changed ones in shared
//           memory, and each entry's new position follows from binary searches
//           (phase_merge).  More changed (a body that turns or deforms), or there is no
//           last list and the body is small: splitters cut the keys into buckets that
//           single CTAs sort in shared memory (phase_scatter, phase_bucket_sort).
//           Otherwise, or if a bucket overflows: four stable LSD radix passes over 8-bit
//           digits, tiles claimed in order, decoupled look-back.
//   build   per chunk of up to 512 sorted positions: de-duplication (keep the first triangle
//           of every distinct code, remove_redundant, Utilities.h:35-55; of more than 524,288
//           triangles in a phase before) and a bottom-up
//           radix-tree build fused with the refit: each leaf thread climbs with handshakes
//           in shared memory while both children lie in the chunk; the parent of range
//           [l, r] is the boundary with the longer common prefix (delta(l-1,l)
//           vs delta(r,r+1), delta = clz(a ^ b) as cudaBRT.cu:9-19), the second
//           child to arrive merges both boxes into the identity box
//           (calculateBoudingBox, cudaBRT.cu:166-206) and continues.  Each chunk
//           then publishes a summary for the nodes that span chunks
//   top     one warp per node that spans chunks: its range ends are the nearest
//           boundaries with a smaller delta, its box the union of its leaves'
//           boxes, both read off the chunk summaries
// What bounds it is latency: a body is a few MB, a barrier about 1.3 us and a dependent
// load through L2 about 0.5, so phases are merged where a grid-wide value is not needed
// between them (de-duplication in the build, centroids kept in registers from the boxes to
// the codes, small bodies without the vertex phase), 32-byte records move as one access,
// and the sorts spread over all CTAs.  Kernel time, before and now: 19,584 triangles with
// few changed codes 32 -> 21 us, with most changed (radix passes before) 69 -> 29, without a
// last order 68 -> 32; 327,680 triangles with few changed 107 -> 71.
// Nodes are numbered by their split position; the tree is the same binary radix
// tree processInternalNode (cudaBRT.cu:120-161) builds, and visg_export_lbvh
// renumbers it into the reference's layout.  Data one CTA reads after another wrote
// it in the same launch is loaded through L2 (ld.global.cg), never the read-only
// path.  Every wait is bounded; a wait that gives up sets ERR_TIMEOUT, the CTA skips
// the rest of its work (still arriving at each barrier), and the host reports
// VISG_ERR_TIMEOUT.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <mutex>

#include "visg_internal.cuh"

namespace visg {

namespace {

constexpr int RB = 512;        // threads per CTA: one chunk of leaves at most, one leaf per thread
constexpr int RW = RB / 32;    // warps per CTA
constexpr int SORT_ITEMS = 4;
constexpr int SORT_TILE = RB * SORT_ITEMS;  // 2048 keys per radix tile
constexpr int RADIX = 256;
constexpr int PASSES = 4;
constexpr int SPREAD_CTAS = 152;    // CTAs a small body is spread over (one per SM)
constexpr int DIRECT_MAX = 65536;   // triangles up to which boxes gather the caller's vertices themselves
constexpr int CHG_CAP = 256;   // changed codes the incremental sort merges (each CTA ranks them all)
constexpr int BK_TARGET = 128; // triangles a bucket of the bucket sort should hold at least
constexpr int BK_CAP = 512;    // and can hold: one key per thread of the sorting CTA
constexpr int BK_MAX = 2048;   // buckets at most
constexpr int OVERSAMPLE = 8;  // keys sampled per bucket for the splitters when there is no last order
constexpr int SAMPLES = 2048;  // and in all
constexpr int SAMPLED_MAX = SAMPLES / OVERSAMPLE * BK_TARGET;  // triangles up to which that is enough
constexpr uint32_t ST_AGG = 1u << 30;
constexpr uint32_t ST_PREFIX = 2u << 30;
constexpr uint32_t ST_VALUE = (1u << 30) - 1u;
constexpr uint32_t CNT_READY = 1u << 31;  // a chunk's leaf count has been published
constexpr int SPIN_LIMIT = 1 << 22;
constexpr uint64_t kGridWaitNs = 1000000000ull;  // a grid barrier gives up after 1 s
constexpr int TOP_STAGED = 1024;  // chunks whose summaries the spanning-node phase stages in shared memory
constexpr int BIG_DELTA = 64;  // above every delta: a boundary that does not exist

__device__ __forceinline__ uint32_t ld_volatile(const uint32_t* p) {
    return *reinterpret_cast<const volatile uint32_t*>(p);
}
__device__ __forceinline__ void st_volatile(uint32_t* p, uint32_t v) { *reinterpret_cast<volatile uint32_t*>(p) = v; }
__device__ __forceinline__ uint64_t now_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Decoupled look-back: the exclusive prefix of tile `tile` from the status words of
// the tiles before it (tile t's at st0[t * stride]: 0 = not yet published, ST_AGG |
// its own count, ST_PREFIX | its inclusive prefix).  A word only ever goes from 0 to
// AGG to PREFIX, so one read of it stays valid: LB_WINDOW predecessors are read per
// round trip, summed in order down to the first PREFIX; a word still 0 is waited on
// (bounded) and the walk resumes there.
constexpr int LB_WINDOW = 8;
__device__ __forceinline__ uint32_t look_back(const uint32_t* st0, size_t stride, int tile, int* err) {
    uint32_t excl = 0;
    int t = tile - 1, spins = 0;
    while (t >= 0) {
        uint32_t w[LB_WINDOW];
#pragma unroll
        for (int q = 0; q < LB_WINDOW; ++q) w[q] = t - q >= 0 ? ld_volatile(st0 + (size_t)(t - q) * stride) : 0u;
        int q = 0;
        bool done = false;
        for (; q < LB_WINDOW && t - q >= 0; ++q) {
            const uint32_t f = w[q] & ~ST_VALUE;
            if (f == 0u) break;  // not published yet
            excl += w[q] & ST_VALUE;
            if (f == ST_PREFIX) {
                done = true;
                break;
            }
        }
        if (done) break;
        t -= q;
        if (q < LB_WINDOW) {  // stopped at an unpublished tile (tile 0 always publishes a PREFIX)
            if (++spins > SPIN_LIMIT) {
                atomicOr(err, ERR_TIMEOUT);
                break;
            }
            __nanosleep(32);
        }
    }
    return excl;
}

// inclusive scan of one value per thread over the CTA (s_warp: 32 words); the CTA
// total is left in s_warp[RW - 1]
__device__ __forceinline__ uint32_t block_scan_incl(uint32_t v, uint32_t* s_warp) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    if (lane == 31) s_warp[warp] = v;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < RW ? s_warp[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t t = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += t;
        }
        if (lane < RW) s_warp[lane] = w;
    }
    __syncthreads();
    uint32_t r = v + (warp > 0 ? s_warp[warp - 1] : 0u);
    __syncthreads();
    return r;
}

// ---- arguments and shared memory ------------------------------------------------------------
struct ChunkView {  // summaries of the chunks (build_chunk)
    int* cmin;
    float4* cbox;
    int2* srec;
    float4* sbox;
    int2* prec;
    float4* pbox;
    uint32_t* rcnt;  // 2 per chunk
    int2* top;
    int* gmin;       // per 32 chunks, for bodies of more than TOP_STAGED chunks: min delta
    float4* gbox;    // and box union (2)
};

struct RebuildArgs {
    const float* xyz;
    const float* nrm;  // null: no thickness push
    const uint32_t* tris;
    int nv, nt;
    float thickness, depth;
    int coherent;  // the last build's sorted list and codes may be reused
    int direct;    // triangles gather the caller's vertices (else the pushed float4 copies)
    int tiles_sort;
    float4* verts;
    float4* tri_box;
    float4* tri_leaf;
    uint32_t* codes;
    uint32_t* keys[2];
    uint32_t* vals[2];
    uint32_t* ucode;
    uint32_t* utri;
    Node* nodes;
    float4* leaves;
    int2* range;
    BvhRoot* root;
    ChunkView cv;
    uint32_t* ghist;   // PASSES x RADIX digit counts
    uint32_t* sstat;   // PASSES x tiles_sort x RADIX look-back status words
    uint32_t* scount;  // PASSES tile counters
    uint32_t* bcnt;    // BK_MAX bucket counts
    unsigned long long* bkey;  // SAMPLES sampled keys in order
    unsigned long long* bslot;  // BK_CAP keys per bucket
    int buckets;               // 0: too many triangles for the bucket sort
    float* part;       // 8 per CTA: its box union (min xyz, max xyz)
    uint32_t* ucnt;    // per chunk: its leaves, with CNT_READY once known
    uint32_t* chg;     // [0] changed codes, then {triangle, new code, old code} x CHG_CAP
    uint32_t* sync;    // [0] barrier arrivals, [1] CTAs finished (both 0 between launches)
    int chunks, chunk_len;
    int* err;
    float4* margin_state;  // cloth records whose query-cache margins the moved body voids
    int64_t m0, m1;        // (vertices [m0, m1): their margin words are cleared)
};

constexpr int MAX_PIECES = 64;  // subtrees a chunk leaves unjoined: at most 31 + 31 + 1 (30-bit codes)
struct BuildSmem {
    // per node and side (A, B): lo (w = link), hi (w = far_end)
    float4 lo[RB][2], hi[RB][2];
    uint32_t flag[RB];      // bit 0: child A arrived, bit 1: child B
    uint32_t code[RB + 2];  // code of position p at p - p0 + 1
    uint32_t lcode[RB], ltri[RB];  // the chunk's leaves, when some position is none
    int delta[RB + 4];      // delta of local boundary j at j + 1
    uint32_t next[32];      // codes after the chunk
    uint32_t wcnt[RW], wsum[RW], pbits[RW];
    float plo[MAX_PIECES][3], phi[MAX_PIECES][3];
    int pend[MAX_PIECES];   // last leaf of each piece
};
static_assert(TOP_STAGED == 2 * RB, "a thread stages the counts of two chunks");
struct TopSmem {
    alignas(8) uint32_t rcnt[2 * TOP_STAGED];
    float lo[TOP_STAGED][3], hi[TOP_STAGED][3];
    int cmin[TOP_STAGED];
    uint32_t pre[TOP_STAGED + 1];
};
struct BucketSmem {
    unsigned long long key[BK_MAX];  // samples, splitters, then the keys of the bucket being sorted
    uint32_t cnt[BK_MAX], base[BK_MAX];
    uint32_t rank[BK_CAP];
};
static_assert(SAMPLES <= BK_MAX, "the samples share the splitters' array");
struct SortSmem {
    uint32_t whist[RW][RADIX + 1];
    uint32_t tstart[RADIX];
    uint32_t gbase[RADIX];
    uint32_t keys[SORT_TILE];
    uint32_t vals[SORT_TILE];
};
struct MergeSmem {
    unsigned long long knew[CHG_CAP];  // changed entries by (new code, triangle)
    unsigned long long kold[CHG_CAP];  // the same entries by (old code, triangle)
    unsigned long long in[2][CHG_CAP];  // both, as they were listed
    uint32_t rank[2][CHG_CAP];
};
constexpr size_t smax(size_t a, size_t b) { return a > b ? a : b; }
constexpr size_t kSmemBytes =
    smax(smax(sizeof(BuildSmem), sizeof(TopSmem)), smax(smax(sizeof(SortSmem), sizeof(MergeSmem)), sizeof(BucketSmem)));

// ---- grid barrier ---------------------------------------------------------------------------
// Every CTA arrives on sync[0] and waits until it holds `target` (gridDim.x per
// barrier so far).  A CTA whose earlier wait gave up (ok false) still arrives, so
// the others are not held, but does not wait.  Returns whether this CTA may go on.
// One thread arrives with a release (cumulative over what the CTA barrier before it
// ordered) and polls with acquires, without sleeping between them.  A barrier of 152 CTAs
// takes 1.2-1.5 us (1.6 with fences around an atomic and 64 ns sleeps).
__device__ bool grid_barrier(uint32_t* ctr, uint32_t& target, bool ok, int* err, int* s_ok) {
    __syncthreads();
    target += gridDim.x;
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(ctr) : "memory");
        int good = ok ? 1 : 0;
        uint64_t t0 = 0;
        for (int polls = 0; good; ++polls) {
            uint32_t v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(ctr) : "memory");
            if (v >= target) break;
            if ((polls & 63) == 63) {
                const uint64_t t = now_ns();
                if (t0 == 0) t0 = t;
                if (t - t0 > kGridWaitNs) {
                    atomicOr(err, ERR_TIMEOUT);
                    good = 0;
                }
            }
        }
        *s_ok = good;
    }
    __syncthreads();
    return *s_ok != 0;
}

// ---- boxes ------------------------------------------------------------------------------------
__device__ __forceinline__ f3 pushed(const RebuildArgs& A, uint32_t v) {  // vertex_extend
    float x = __ldg(A.xyz + 3 * v), y = __ldg(A.xyz + 3 * v + 1), z = __ldg(A.xyz + 3 * v + 2);
    if (A.nrm) {
        x = __fadd_rn(x, __fmul_rn(A.thickness, __ldg(A.nrm + 3 * v)));
        y = __fadd_rn(y, __fmul_rn(A.thickness, __ldg(A.nrm + 3 * v + 1)));
        z = __fadd_rn(z, __fmul_rn(A.thickness, __ldg(A.nrm + 3 * v + 2)));
    }
    return mk3(x, y, z);
}

__device__ __forceinline__ void box_add(f3& lo, f3& hi, f3 p) {
    lo.x = fminf(lo.x, p.x); lo.y = fminf(lo.y, p.y); lo.z = fminf(lo.z, p.z);
    hi.x = fmaxf(hi.x, p.x); hi.y = fmaxf(hi.y, p.y); hi.z = fmaxf(hi.z, p.z);
}

// min (k < 3) / max (k >= 3) of r[6] over the CTA, into s_red[6] (all threads)
__device__ __forceinline__ void block_box_reduce(float r[6], float* s_red /* 6 * RW */) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int k = 0; k < 3; ++k) r[k] = fminf(r[k], __shfl_xor_sync(0xffffffffu, r[k], o));
#pragma unroll
        for (int k = 3; k < 6; ++k) r[k] = fmaxf(r[k], __shfl_xor_sync(0xffffffffu, r[k], o));
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0)
        for (int k = 0; k < 6; ++k) s_red[k * RW + warp] = r[k];
    __syncthreads();
    if (warp < 6) {  // warp k: component k of all warps
        float v = s_red[warp * RW + (lane & (RW - 1))];
#pragma unroll
        for (int o = RW / 2; o > 0; o >>= 1) {
            const float w = __shfl_xor_sync(0xffffffffu, v, o);
            v = warp < 3 ? fminf(v, w) : fmaxf(v, w);
        }
        if (lane == 0) s_red[warp * RW] = v;
    }
    __syncthreads();
}

// the pushed vertices, as float4 (one aligned load per corner in phase_boxes); the
// query-cache margins of the body's cloth vertices are voided (the body moves)
__device__ void phase_verts(const RebuildArgs& A) {
    for (int v = blockIdx.x * RB + threadIdx.x; v < A.nv; v += gridDim.x * RB) {
        const f3 p = pushed(A, (uint32_t)v);
        A.verts[v] = make_float4(p.x, p.y, p.z, 0.0f);
    }
    if (A.margin_state)
        for (int64_t i = A.m0 + (int64_t)blockIdx.x * RB + threadIdx.x; i < A.m1; i += (int64_t)gridDim.x * RB)
            reinterpret_cast<float*>(A.margin_state + rec_at(i) + 32)[3] = 0.0f;
}

constexpr int BOX_BATCH = 3;  // triangles a thread loads before it computes any

// each triangle's expanded box (BBox(v0).expand(v1).expand(v2) and the three
// corners pushed inward by depth * n) and leaf record; the CTA's union of its boxes
// with the identity box in part[8 * cta].  The centroids of a thread's first BOX_BATCH
// triangles stay in its registers: phase_codes takes the same triangles.
template <bool DIRECT>
__device__ void phase_boxes(const RebuildArgs& A, float* s_red, f3 (&cen)[BOX_BATCH]) {
    const int stride = gridDim.x * RB;
    const int first = blockIdx.x * RB + threadIdx.x;
    f3 lo = mk3(100.0f, 100.0f, 100.0f), hi = mk3(-100.0f, -100.0f, -100.0f);
    for (int base = first; base < A.nt; base += BOX_BATCH * stride) {
        uint32_t idx[BOX_BATCH][3];
#pragma unroll
        for (int q = 0; q < BOX_BATCH; ++q) {
            const int t = base + q * stride;
#pragma unroll
            for (int c = 0; c < 3; ++c) idx[q][c] = t < A.nt ? __ldg(A.tris + 3 * t + c) : 0u;
        }
        f3 w[BOX_BATCH][3];
#pragma unroll
        for (int q = 0; q < BOX_BATCH; ++q)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                // vertex indices come from the caller: one out of range is recorded and
                // read as vertex 0, so no load leaves the vertex array (the build's
                // result is then reported as failed)
                uint32_t v = idx[q][c];
                if (v >= (uint32_t)A.nv) {
                    if (base + q * stride < A.nt) atomicOr(A.err, ERR_INDEX);
                    v = 0u;
                }
                w[q][c] = DIRECT ? pushed(A, v) : xyz(__ldcg(A.verts + v));
            }
#pragma unroll
        for (int q = 0; q < BOX_BATCH; ++q) {
            const int t = base + q * stride;
            if (t >= A.nt) break;
            const f3 v0 = w[q][0], v1 = w[q][1], v2 = w[q][2];
            const f3 n = normalize(cross(sub(v1, v0), sub(v2, v0)));  // Primitive::d_get_normal
            f3 blo = v0, bhi = v0;
            box_add(blo, bhi, v1);
            box_add(blo, bhi, v2);
            const f3 dn = mul(A.depth, n);
            box_add(blo, bhi, sub(v0, dn));
            box_add(blo, bhi, sub(v1, dn));
            box_add(blo, bhi, sub(v2, dn));
            st8(A.tri_box + 2 * t, make_float4(blo.x, blo.y, blo.z, 0.0f), make_float4(bhi.x, bhi.y, bhi.z, 0.0f));
            st8(A.tri_leaf + 2 * t, make_float4(v0.x, v0.y, v0.z, n.x),
                make_float4(n.y, n.z, __int_as_float(t), 0.0f));
            box_add(lo, hi, blo);
            box_add(lo, hi, bhi);
            if (base == first) cen[q] = divs(add(blo, bhi), 2.0f);  // BBox::centroid
        }
    }
    float r[6] = {lo.x, lo.y, lo.z, hi.x, hi.y, hi.z};
    block_box_reduce(r, s_red);
    if (threadIdx.x < 6) A.part[8 * blockIdx.x + threadIdx.x] = s_red[threadIdx.x * RW];
}

// ---- codes ------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t expand_bits(uint32_t v) {  // bvh.cu:20-27
    v = (v * 0x00010001u) & 0xFF0000FFu;
    v = (v * 0x00000101u) & 0x0F00F00Fu;
    v = (v * 0x00000011u) & 0xC30C30C3u;
    v = (v * 0x00000005u) & 0x49249249u;
    return v;
}

// the frame from the CTA unions; each triangle's code; with `listing`, the triangles
// whose code changed go to the change list (at most CHG_CAP are stored)
__device__ void phase_codes(const RebuildArgs& A, bool listing, float* s_red, float* s_frame, f3 (&cen)[BOX_BATCH],
                            uint32_t (&old)[BOX_BATCH]) {
    float r[6] = {100.0f, 100.0f, 100.0f, -100.0f, -100.0f, -100.0f};
    for (int c = threadIdx.x; c < (int)gridDim.x; c += RB) {
#pragma unroll
        for (int k = 0; k < 3; ++k) r[k] = fminf(r[k], __ldcg(A.part + 8 * c + k));
#pragma unroll
        for (int k = 3; k < 6; ++k) r[k] = fmaxf(r[k], __ldcg(A.part + 8 * c + k));
    }
    block_box_reduce(r, s_red);
    if (threadIdx.x < 6) s_frame[threadIdx.x] = s_red[threadIdx.x * RW];
    __syncthreads();
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        A.root->frame_lo = make_float4(s_frame[0], s_frame[1], s_frame[2], 0.0f);
        A.root->frame_hi = make_float4(s_frame[3], s_frame[4], s_frame[5], 0.0f);
    }
    const f3 fmn = mk3(s_frame[0], s_frame[1], s_frame[2]);
    const f3 ext = sub(mk3(s_frame[3], s_frame[4], s_frame[5]), fmn);
    const bool flat = length(ext) == 0.0f;
    const int lane = threadIdx.x & 31;
    const int stride = gridDim.x * RB;
    const int first = blockIdx.x * RB;
    for (int base = first; base < A.nt; base += BOX_BATCH * stride) {  // warp-uniform bounds
        // all triangles' loads first
        if (base != first)
#pragma unroll
            for (int q = 0; q < BOX_BATCH; ++q) {
                const int t = base + q * stride + threadIdx.x;
                if (t < A.nt) {
                    const f4x2 b = ld8_cg(A.tri_box + 2 * t);
                    cen[q] = divs(add(xyz(b.a), xyz(b.b)), 2.0f);
                    if (listing) old[q] = A.codes[t];
                }
            }
#pragma unroll
        for (int q = 0; q < BOX_BATCH; ++q) {
            const int t = base + q * stride + threadIdx.x;
            if (base + q * stride >= A.nt) break;
            bool changed = false;
            uint32_t code = 0u;
            if (t < A.nt) {
                const f3 c = cen[q];
                f3 u = mk3(0.0f, 0.0f, 0.0f);
                if (!flat) u = divv(sub(c, fmn), ext);  // BBox::getUnitcubePosOf
                const float x = fminf(fmaxf(__fmul_rn(u.x, 1024.0f), 0.0f), 1023.0f);
                const float y = fminf(fmaxf(__fmul_rn(u.y, 1024.0f), 0.0f), 1023.0f);
                const float z = fminf(fmaxf(__fmul_rn(u.z, 1024.0f), 0.0f), 1023.0f);
                code = expand_bits((uint32_t)x) * 4u + expand_bits((uint32_t)y) * 2u + expand_bits((uint32_t)z);
                A.codes[t] = code;
                changed = listing && old[q] != code;
            }
            const unsigned m = __ballot_sync(0xffffffffu, changed);
            if (m) {
                const int leader = __ffs(m) - 1;
                uint32_t b0 = 0;
                if (lane == leader) b0 = atomicAdd(A.chg, (uint32_t)__popc(m));
                b0 = __shfl_sync(0xffffffffu, b0, leader);
                const uint32_t k = b0 + (uint32_t)__popc(m & ((1u << lane) - 1u));
                if (changed && k < (uint32_t)CHG_CAP) {
                    A.chg[1 + 3 * k] = (uint32_t)t;
                    A.chg[2 + 3 * k] = code;
                    A.chg[3 + 3 * k] = old[q];
                }
            }
        }
    }
}

// ---- sort: incremental merge --------------------------------------------------------------------
__device__ __forceinline__ unsigned long long key64(uint32_t code, uint32_t tri) {
    return ((unsigned long long)code << 32) | tri;
}
// entries of a[0, n) below x (a ascending)
__device__ __forceinline__ int lower_bound64(const unsigned long long* a, int n, unsigned long long x) {
    int lo = 0, len = n;
    while (len > 0) {
        const int h = len >> 1;
        if (a[lo + h] < x) {
            lo += h + 1;
            len -= h + 1;
        } else {
            len = h;
        }
    }
    return lo;
}

// rank[i] += the keys of a[0, n) below a[i] (distinct keys, n <= RB, rank zero before), by
// comparing all pairs: the CTA's threads share out n rows and, for a short list, parts of
// the columns.  For the few hundred keys it is used on this takes a third of the time of
// a bitonic sort, whose stages are all exchange: 128 keys 0.3 us.
__device__ __forceinline__ void rank_keys(const unsigned long long* a, int n, uint32_t* rank) {
    int rows = 32;
    while (rows < n) rows <<= 1;  // at most RB
    const int parts = RB / rows, part = (int)threadIdx.x / rows, i = (int)threadIdx.x & (rows - 1);
    if (i < n) {
        const unsigned long long x = a[i];
        const int j1 = (part + 1) * n / parts;
        uint32_t r = 0;
#pragma unroll 8
        for (int j = part * n / parts; j < j1; ++j) r += a[j] < x ? 1u : 0u;
        atomicAdd(&rank[i], r);
    }
}

// Merge of the nc changed entries into the last build's sorted list ko/vo (all nt
// triangles by (code, triangle), old codes): every CTA sorts the changed entries by
// new key (knew) and by old key (kold), then walks its slice of the old list.  For
// old slot s with key k_s, q(s) = #kold < k_s and r(s) = #knew < k_s.  An unchanged
// entry keeps its code, so its key is k_s and its new position is s - q(s) (the
// unchanged entries before it) + r(s) (the changed entries that now sort before
// it).  Changed entry j with r(s) <= j < r(s + 1) lies strictly between k_s and
// k_(s+1): s + 1 - q(s + 1) unchanged entries sort before it, j changed ones, so its
// position is j + s + 1 - q(s + 1).  Changed entries below the first old key go to
// positions j (CTA 0).  Positions are a permutation of [0, nt); each is checked.
__device__ void phase_merge(const RebuildArgs& A, int nc, const uint32_t* ko, const uint32_t* vo, uint32_t* kn,
                            uint32_t* vn, MergeSmem& S) {
    for (int k = threadIdx.x; k < nc; k += RB) {
        const uint32_t t = __ldcg(A.chg + 1 + 3 * k);
        S.in[0][k] = key64(__ldcg(A.chg + 2 + 3 * k), t);
        S.in[1][k] = key64(__ldcg(A.chg + 3 + 3 * k), t);
        S.rank[0][k] = S.rank[1][k] = 0u;
    }
    __syncthreads();
    rank_keys(S.in[0], nc, S.rank[0]);
    rank_keys(S.in[1], nc, S.rank[1]);
    __syncthreads();
    for (int k = threadIdx.x; k < nc; k += RB) {
        S.knew[S.rank[0][k]] = S.in[0][k];
        S.kold[S.rank[1][k]] = S.in[1][k];
    }
    __syncthreads();
    const int nt = A.nt;
    const int per = (nt + gridDim.x - 1) / gridDim.x;
    const int a = blockIdx.x * per, b = min(nt, a + per);
    constexpr int MB = 3;  // slots a thread loads before it searches
    const int lane = (int)(threadIdx.x & 31u);
    for (int w0 = a + ((int)threadIdx.x & ~31); w0 < b; w0 += MB * RB) {  // warp-uniform
        unsigned long long ks[MB];
#pragma unroll
        for (int u = 0; u < MB; ++u) {  // lane 31's next slot is searched for by nobody else: load it too
            const int s = w0 + u * RB + lane;
            ks[u] = s < nt ? key64(ko[s], vo[s]) : ~0ull;
        }
        unsigned long long kx[MB];
#pragma unroll
        for (int u = 0; u < MB; ++u) {
            const int s = w0 + u * RB + 32;
            kx[u] = lane == 31 && s < nt ? key64(ko[s], vo[s]) : ~0ull;
        }
#pragma unroll
        for (int u = 0; u < MB; ++u) {
            const int s = w0 + u * RB + lane;
            const int q = lower_bound64(S.kold, nc, ks[u]), r = lower_bound64(S.knew, nc, ks[u]);
            // the next slot's counts: the next lane's
            int q1 = __shfl_down_sync(0xffffffffu, q, 1), r1 = __shfl_down_sync(0xffffffffu, r, 1);
            if (lane == 31) {
                q1 = lower_bound64(S.kold, nc, kx[u]);
                r1 = lower_bound64(S.knew, nc, kx[u]);
            }
            if (s >= b) continue;
            if (!(q < nc && S.kold[q] == ks[u])) {  // unchanged
                const int pos = s - q + r;
                if ((unsigned)pos < (unsigned)nt) {
                    kn[pos] = (uint32_t)(ks[u] >> 32);
                    vn[pos] = (uint32_t)ks[u];
                }
            }
            for (int j = r; j < r1; ++j) {
                const int pos = j + s + 1 - q1;
                if ((unsigned)pos < (unsigned)nt) {
                    kn[pos] = (uint32_t)(S.knew[j] >> 32);
                    vn[pos] = (uint32_t)S.knew[j];
                }
            }
        }
    }
    if (blockIdx.x == 0 && nt > 0) {
        const int r0 = lower_bound64(S.knew, nc, key64(ko[0], vo[0]));
        for (int j = threadIdx.x; j < r0; j += RB) {
            kn[j] = (uint32_t)(S.knew[j] >> 32);
            vn[j] = (uint32_t)S.knew[j];
        }
    }
}

// ---- sort: buckets -------------------------------------------------------------------------------
// Too many codes changed for a merge (an animated body): splitters cut the keys (code,
// triangle) into nb buckets of at least about BK_TARGET; phase_scatter puts every
// triangle's key into its bucket's slots (in any order), and after a grid barrier each
// bucket is sorted by one CTA in shared memory (phase_bucket_sort).  The splitters are
// nb - 1 entries at equal distances of the last build's list, whose codes have moved only
// a little; without one, of a sample.  The keys are distinct, so equal codes do not fill a
// bucket.  Small buckets, so that a small body's sort takes all SMs.  The slots are an array
// of their own: a build that gives up after phase_scatter leaves whatever it wrote, and
// the steps behind it in the stream still walk the nodes, whose links must be in range.
//
// The i-th of ns sampled triangles: one from each of ns equal parts of the list, at a
// scrambled place in its part (a mesh's rows repeat: at equal distances the sample of the
// capsules fell on the same few angles of every ring).
__device__ __forceinline__ uint32_t sampled(int i, int ns, int nt) {
    const int64_t t = (int64_t)i * nt / ns, len = (int64_t)(i + 1) * nt / ns - t;
    return (uint32_t)(t + (len > 1 ? (int64_t)(((uint32_t)i * 2654435761u) >> 8) % len : 0));
}

// phase_sample: the CTAs rank the sampled keys among themselves, each its share, and
// leave them in order in A.bkey.
__device__ void phase_sample(const RebuildArgs& A, int ns, BucketSmem& S) {
    for (int i = threadIdx.x; i < ns; i += RB) {
        S.key[i] = key64(__ldcg(A.codes + sampled(i, ns, A.nt)), (uint32_t)i);  // by (code, place): distinct
    }
    __syncthreads();
    const int lane = (int)(threadIdx.x & 31u);
    for (int i = blockIdx.x * RW + (int)(threadIdx.x >> 5); i < ns; i += gridDim.x * RW) {
        const unsigned long long x = S.key[i];
        uint32_t r = 0;
#pragma unroll 8
        for (int j = lane; j < ns; j += 32) r += S.key[j] < x ? 1u : 0u;
        r = __reduce_add_sync(0xffffffffu, r);
        if (lane == 0) A.bkey[r] = key64((uint32_t)(x >> 32), sampled(i, ns, A.nt));
    }
}

__device__ void phase_scatter(const RebuildArgs& A, int nb, const uint32_t* ko, const uint32_t* vo, BucketSmem& S) {
    const int nt = A.nt;
    for (int i = threadIdx.x; i < nb - 1; i += RB) {
        if (ko) {
            const int p = (int)((int64_t)(i + 1) * nt / nb);
            S.key[i] = key64(ko[p], vo[p]);
        } else {
            S.key[i] = __ldcg(A.bkey + (i + 1) * OVERSAMPLE);
        }
    }
    unsigned long long* const slots = A.bslot;
    const int per = (nt + gridDim.x - 1) / gridDim.x;
    const int a = blockIdx.x * per, b = min(nt, a + per);
    constexpr int ITEMS = 4;
    for (int s0 = a; s0 < b; s0 += ITEMS * RB) {
        for (int k = threadIdx.x; k < nb; k += RB) S.cnt[k] = 0u;
        __syncthreads();
        unsigned long long key[ITEMS];
        uint32_t rank[ITEMS];
        int bk[ITEMS];
#pragma unroll
        for (int u = 0; u < ITEMS; ++u) {
            const int t = s0 + u * RB + threadIdx.x;
            key[u] = t < b ? key64(__ldcg(A.codes + t), (uint32_t)t) : ~0ull;
        }
#pragma unroll
        for (int u = 0; u < ITEMS; ++u)
            if (key[u] != ~0ull) {
                bk[u] = lower_bound64(S.key, nb - 1, key[u] + 1ull);  // splitters <= key
                rank[u] = atomicAdd(&S.cnt[bk[u]], 1u);
            }
        __syncthreads();
        for (int k = threadIdx.x; k < nb; k += RB)
            if (S.cnt[k]) S.base[k] = atomicAdd(A.bcnt + k, S.cnt[k]);
        __syncthreads();
#pragma unroll
        for (int u = 0; u < ITEMS; ++u)
            if (key[u] != ~0ull) {
                const uint32_t pos = S.base[bk[u]] + rank[u];
                if (pos < (uint32_t)BK_CAP) slots[(size_t)bk[u] * BK_CAP + pos] = key[u];  // else: see buckets_fit
            }
        __syncthreads();
    }
}

// whether no bucket was given more than it holds (the same answer in every CTA); S.cnt
// then holds the counts and S.base the places of the buckets in the sorted list
__device__ bool buckets_fit(const RebuildArgs& A, int nb, BucketSmem& S, uint32_t* s_scan) {
    constexpr int E = BK_MAX / RB;
    uint32_t c[E], sum = 0;
    bool over = false;
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int i = E * (int)threadIdx.x + e;
        c[e] = i < nb ? __ldcg(A.bcnt + i) : 0u;
        sum += c[e];
        over |= c[e] > (uint32_t)BK_CAP;
    }
    uint32_t off = block_scan_incl(sum, s_scan) - sum;
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int i = E * (int)threadIdx.x + e;
        S.cnt[i] = c[e];
        S.base[i] = off;
        off += c[e];
    }
    return __syncthreads_or(over ? 1 : 0) == 0;
}

__device__ void phase_bucket_sort(const RebuildArgs& A, int nb, uint32_t* kn, uint32_t* vn, BucketSmem& S) {
    const unsigned long long* const slots = A.bslot;
    const int i = (int)threadIdx.x;
    for (int b = blockIdx.x; b < nb; b += gridDim.x) {
        const int n = (int)S.cnt[b];
        const uint32_t off = S.base[b];
        const unsigned long long k = i < n ? __ldcg(slots + (size_t)b * BK_CAP + i) : 0ull;
        S.rank[i] = 0u;
        if (i < n) S.key[i] = k;
        __syncthreads();
        rank_keys(S.key, n, S.rank);
        __syncthreads();
        if (i < n) {
            const uint32_t o = off + S.rank[i];
            if (o < (uint32_t)A.nt) {
                kn[o] = (uint32_t)(k >> 32);
                vn[o] = (uint32_t)k;
            }
        }
    }
}

// ---- sort: radix passes ------------------------------------------------------------------------
// digit counts of all four passes (grid-stride over the codes, per CTA in shared memory)
__device__ void phase_hist(const RebuildArgs& A, uint32_t* s_hist /* PASSES * RADIX */) {
    for (int k = threadIdx.x; k < PASSES * RADIX; k += RB) s_hist[k] = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    for (int base = blockIdx.x * RB; base < A.nt; base += gridDim.x * RB) {
        const int t = base + threadIdx.x;
        const bool ok = t < A.nt;
        const uint32_t code = ok ? __ldcg(A.codes + t) : 0u;
        // the two high digits are nearly constant across neighbouring triangles, so
        // their lanes add once per equal digit
#pragma unroll
        for (int p = 0; p < PASSES; ++p) {
            const uint32_t dig = (code >> (8 * p)) & 255u;
            if (p < 2) {
                if (ok) atomicAdd(&s_hist[p * RADIX + dig], 1u);
            } else {
                const uint32_t peers = __match_any_sync(0xffffffffu, ok ? dig : RADIX);
                if (ok && lane == __ffs(peers) - 1) atomicAdd(&s_hist[p * RADIX + dig], (uint32_t)__popc(peers));
            }
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < PASSES * RADIX; k += RB) {
        const uint32_t v = s_hist[k];
        if (v) atomicAdd(&A.ghist[k], v);
    }
}

// One tile of a stable LSD pass over 8-bit digit (key >> shift) & 255.  Tiles are
// claimed in order through a counter, so every tile a CTA waits on belongs to a CTA
// that is already at work on it: the look-back always terminates.
__device__ void sort_tile(const uint32_t* kin, const uint32_t* vin, uint32_t* kout, uint32_t* vout, int n, int shift,
                          const uint32_t* ghist, uint32_t* status, int tile, SortSmem& S, uint32_t* s_scan, int* err) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int k = tid; k < RW * (RADIX + 1); k += RB) (&S.whist[0][0])[k] = 0;
    __syncthreads();
    const int base = tile * SORT_TILE + warp * (32 * SORT_ITEMS);
    uint32_t key[SORT_ITEMS], val[SORT_ITEMS], rank[SORT_ITEMS];
    int dig[SORT_ITEMS];
#pragma unroll
    for (int j = 0; j < SORT_ITEMS; ++j) {
        const int idx = base + j * 32 + lane;  // warp-striped: j-major order is input order
        if (idx < n) {
            key[j] = __ldcg(kin + idx);
            val[j] = vin ? __ldcg(vin + idx) : (uint32_t)idx;
            dig[j] = (int)((key[j] >> shift) & 255u);
        } else {
            key[j] = 0u;
            val[j] = 0u;
            dig[j] = RADIX;  // padding: own bucket, never written
        }
    }
    // stable rank of every key among equal digits of this warp, in input order
#pragma unroll
    for (int j = 0; j < SORT_ITEMS; ++j) {
        const uint32_t peers = __match_any_sync(0xffffffffu, dig[j]);
        const int leader = __ffs(peers) - 1;
        uint32_t before = 0;
        if (lane == leader) {
            before = S.whist[warp][dig[j]];
            S.whist[warp][dig[j]] = before + __popc(peers);
        }
        before = __shfl_sync(0xffffffffu, before, leader);
        rank[j] = before + __popc(peers & ((1u << lane) - 1u));
        __syncwarp();
    }
    __syncthreads();
    // thread d < RADIX owns digit d: warp-exclusive prefixes and the tile count
    const int d = tid;
    uint32_t tcount = 0;
    if (d < RADIX) {
        uint32_t run = 0;
#pragma unroll
        for (int w = 0; w < RW; ++w) {
            const uint32_t c = S.whist[w][d];
            S.whist[w][d] = run;
            run += c;
        }
        tcount = run;
    }
    const uint32_t tincl = block_scan_incl(tcount, s_scan);
    if (d < RADIX) S.tstart[d] = tincl - tcount;
    const uint32_t gh = d < RADIX ? __ldcg(ghist + d) : 0u;
    const uint32_t goff = block_scan_incl(gh, s_scan) - gh;
    // publish the tile's count of digit d, then look back for the exclusive prefix
    if (d < RADIX) {
        uint32_t excl = 0;
        uint32_t* st = status + (size_t)tile * RADIX + d;
        if (tile == 0) {
            st_volatile(st, ST_PREFIX | tcount);
        } else {
            st_volatile(st, ST_AGG | tcount);
            excl = look_back(status + d, RADIX, tile, err);
            st_volatile(st, ST_PREFIX | ((excl + tcount) & ST_VALUE));
        }
        S.gbase[d] = goff + excl;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < SORT_ITEMS; ++j) {
        if (dig[j] < RADIX) {
            const uint32_t pos = S.tstart[dig[j]] + S.whist[warp][dig[j]] + rank[j];
            S.keys[pos] = key[j];
            S.vals[pos] = val[j];
        }
    }
    __syncthreads();
    const int tile_n = min(SORT_TILE, n - tile * SORT_TILE);
    for (int p = tid; p < tile_n; p += RB) {
        const uint32_t k = S.keys[p];
        const uint32_t dd = (k >> shift) & 255u;
        const uint32_t o = S.gbase[dd] + (uint32_t)p - S.tstart[dd];
        if (o < (uint32_t)n) {  // always true unless a look-back gave up
            kout[o] = k;
            vout[o] = S.vals[p];
        }
    }
    __syncthreads();
}

__device__ void phase_sort_pass(const RebuildArgs& A, int p, SortSmem& S, uint32_t* s_scan, int* s_claim) {
    const uint32_t* kin = p == 0 ? A.codes : A.keys[(p - 1) & 1];
    const uint32_t* vin = p == 0 ? nullptr : A.vals[(p - 1) & 1];
    for (;;) {
        if (threadIdx.x == 0) *s_claim = (int)atomicAdd(A.scount + p, 1u);
        __syncthreads();
        const int tile = *s_claim;
        __syncthreads();
        if (tile >= A.tiles_sort) break;
        sort_tile(kin, vin, A.keys[p & 1], A.vals[p & 1], A.nt, 8 * p, A.ghist + p * RADIX,
                  A.sstat + (size_t)p * A.tiles_sort * RADIX, tile, S, s_scan, A.err);
    }
}

// ---- unique (bodies of more than TOP_STAGED chunks) ------------------------------------------------
// De-duplication before the build.  A large body's codes are crowded (10 bits an axis), so many
// triangles share one, and chunks of sorted positions would be chunks of few leaves: 5.1 M
// triangles with 2.4 M codes take 641 us a rebuild with the de-duplication in the build, 362
// with it before; 21.8 M with 4.7 M 2,371 and 966.  CTA c takes the positions [c per, (c + 1) per) of the sorted list.
constexpr int UNIQ_ITEMS = 4;
__device__ __forceinline__ int unique_slice(const RebuildArgs& A, int& b) {
    const int per = (A.nt + (int)gridDim.x - 1) / (int)gridDim.x;
    const int a = (int)min((int64_t)blockIdx.x * per, (int64_t)A.nt);
    b = min(A.nt, a + per);
    return a;
}
// bit j: position p + j step is a leaf (position 0, or its code differs from the one before's)
__device__ __forceinline__ uint32_t leaf_bits(const uint32_t* K, int p, int step, int b, uint32_t (&k)[UNIQ_ITEMS]) {
    uint32_t before[UNIQ_ITEMS], f = 0;
#pragma unroll
    for (int j = 0; j < UNIQ_ITEMS; ++j) {
        const int q = p + j * step;
        k[j] = q < b ? __ldcg(K + q) : 0u;
        before[j] = q < b && q > 0 ? __ldcg(K + q - 1) : 0u;
    }
#pragma unroll
    for (int j = 0; j < UNIQ_ITEMS; ++j)
        if (p + j * step < b && (p + j * step == 0 || k[j] != before[j])) f |= 1u << j;
    return f;
}
__device__ void phase_unique_count(const RebuildArgs& A, const uint32_t* K, uint32_t* s_scan) {
    int b;
    const int a = unique_slice(A, b);
    uint32_t k[UNIQ_ITEMS], c = 0;
    for (int p = a + (int)threadIdx.x; p < b; p += RB * UNIQ_ITEMS) c += __popc(leaf_bits(K, p, RB, b, k));
    block_scan_incl(c, s_scan);
    if (threadIdx.x == 0) A.ucnt[blockIdx.x] = s_scan[RW - 1];
}
// the leaves of this CTA's slice at its offset; returns the number of leaves in all
__device__ int phase_unique_write(const RebuildArgs& A, const uint32_t* K, const uint32_t* V, uint32_t* s_scan) {
    uint32_t before = 0, all = 0;
    for (int c = threadIdx.x; c < (int)gridDim.x; c += RB) {
        const uint32_t v = __ldcg(A.ucnt + c);
        all += v;
        if (c < (int)blockIdx.x) before += v;
    }
    block_scan_incl(before, s_scan);
    uint32_t off = s_scan[RW - 1];
    __syncthreads();
    block_scan_incl(all, s_scan);
    const int n = (int)min(s_scan[RW - 1], (uint32_t)A.nt);
    __syncthreads();
    int b;
    const int a = unique_slice(A, b);
    for (int base = a; base < b; base += RB * UNIQ_ITEMS) {
        const int p = base + (int)threadIdx.x * UNIQ_ITEMS;
        uint32_t k[UNIQ_ITEMS], t[UNIQ_ITEMS];
#pragma unroll
        for (int j = 0; j < UNIQ_ITEMS; ++j) t[j] = p + j < b ? __ldcg(V + p + j) : 0u;
        const uint32_t f = leaf_bits(K, p, 1, b, k), cnt = (uint32_t)__popc(f);
        uint32_t o = off + block_scan_incl(cnt, s_scan) - cnt;
        off += s_scan[RW - 1];
#pragma unroll
        for (int j = 0; j < UNIQ_ITEMS; ++j)
            if (f >> j & 1u) {
                if (o < (uint32_t)A.nt) {
                    A.ucode[o] = k[j];
                    A.utri[o] = t[j];
                }
                ++o;
            }
        __syncthreads();  // s_scan is read above before the next scan overwrites it
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) A.root->n_leaves = n;
    return n;
}

// ---- build ---------------------------------------------------------------------------------------
// identity box (min +100, max -100) expanded by child A then child B
__device__ __forceinline__ void merge_ab(float4 alo, float4 ahi, float4 blo, float4 bhi, float4& lo, float4& hi) {
    lo = make_float4(fminf(fminf(100.0f, alo.x), blo.x), fminf(fminf(100.0f, alo.y), blo.y),
                     fminf(fminf(100.0f, alo.z), blo.z), 0.0f);
    hi = make_float4(fmaxf(fmaxf(-100.0f, ahi.x), bhi.x), fmaxf(fmaxf(-100.0f, ahi.y), bhi.y),
                     fmaxf(fmaxf(-100.0f, ahi.z), bhi.z), 0.0f);
}

// The child (lo, hi, link) over leaves [l, r] enters its parent g: its side of the
// node and of the node's leaf range.
__device__ __forceinline__ void write_side(Node* nodes, int2* range, int g, bool is_a, float4 lo, float4 hi, int link,
                                           int l, int r) {
    st8(is_a ? &nodes[g].a_lo : &nodes[g].b_lo, make_float4(lo.x, lo.y, lo.z, __int_as_float(link)),
        make_float4(hi.x, hi.y, hi.z, 0.0f));
    if (is_a) range[g].x = l;  // leaf ranges of the nodes (read by the export)
    else range[g].y = r;
}

// box union (fminf / fmaxf: exact, so any grouping gives the same box)
__device__ __forceinline__ void box_union(float4& lo, float4& hi, float4 lo2, float4 hi2) {
    lo = make_float4(fminf(lo.x, lo2.x), fminf(lo.y, lo2.y), fminf(lo.z, lo2.z), 0.0f);
    hi = make_float4(fmaxf(hi.x, hi2.x), fmaxf(hi.y, hi2.y), fmaxf(hi.z, hi2.z), 0.0f);
}
__device__ __forceinline__ float4 ident_lo() { return make_float4(100.0f, 100.0f, 100.0f, 0.0f); }
__device__ __forceinline__ float4 ident_hi() { return make_float4(-100.0f, -100.0f, -100.0f, 0.0f); }
__device__ __forceinline__ float4 shfl_f4(float4 v, int o) {  // from the lane o below
    return make_float4(__shfl_up_sync(0xffffffffu, v.x, o), __shfl_up_sync(0xffffffffu, v.y, o),
                       __shfl_up_sync(0xffffffffu, v.z, o), 0.0f);
}
__device__ __forceinline__ void warp_box_reduce(float4& lo, float4& hi) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float4 l2 = make_float4(__shfl_xor_sync(0xffffffffu, lo.x, o), __shfl_xor_sync(0xffffffffu, lo.y, o),
                                      __shfl_xor_sync(0xffffffffu, lo.z, o), 0.0f);
        const float4 h2 = make_float4(__shfl_xor_sync(0xffffffffu, hi.x, o), __shfl_xor_sync(0xffffffffu, hi.y, o),
                                      __shfl_xor_sync(0xffffffffu, hi.z, o), 0.0f);
        box_union(lo, hi, l2, h2);
    }
}

// a child's far range end (a leaf of the chunk) with delta at the boundary beyond it, so
// that the climb need not look the delta up again
__device__ __forceinline__ int far_end(int leaf, int delta) { return leaf | (delta + 1) << 16; }
__device__ __forceinline__ int far_leaf(int w) { return w & 0xffff; }
__device__ __forceinline__ int far_delta(int w) { return (w >> 16) - 1; }

// De-duplication, bottom-up build of the chunk-local nodes, and the chunk summary.  A
// chunk is at most RB positions [p0, p0 + m) of the sorted list (chunk_length); its leaves are the positions
// whose code differs from the one before (remove_redundant, Utilities.h:35-55: the first
// triangle of every code).  The chunk works in its own leaf numbers; where its leaves
// begin in the whole is the sum of the counts that the chunks before it publish, read
// when its climb is done (every CTA publishes a chunk's count before it waits, and takes
// its chunks in ascending order, so every count that is waited for comes).
//
// The climb goes through the nodes split inside the chunk in shared memory only: each
// child leaves its box, link and far range end in its side of the node's slot; the first
// to arrive stops, the second merges (A then B) and climbs on.  Nodes both of whose
// children arrived are written out.  What stays unjoined are pieces: subtrees over
// consecutive leaves whose parent needs another chunk.  A piece's side is written into
// its parent, and the boundaries after the pieces are the nodes that span chunks, which
// phase_top finishes from the summary:
//   * a node elsewhere whose range ends inside this chunk ends at a boundary after a
//     piece (a boundary inside a piece has a larger delta than the piece's ends), so the
//     records are the strict suffix minima of delta over those boundaries (the nearest
//     smaller delta to the left of a node further right) and the strict prefix minima (to
//     the right of a node further left), at most 31 each, with the union of the
//     chunk's leaf boxes beyond / up to each of them;
//   * the chunk's min delta and leaf box union.
// Two warps make the summary of at most 63 pieces, two per lane, from either end.
// BIG: K and V are the np leaves themselves (phase_unique), so a chunk's positions are its
// leaves and their numbers.
template <bool BIG>
__device__ void build_chunk(const RebuildArgs& A, int chunk, int np, const uint32_t* K, const uint32_t* V,
                            BuildSmem& S) {
    const float inf = __int_as_float(0x7f800000);
    const ChunkView& cv = A.cv;
    const int tid = (int)threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int p0 = chunk * A.chunk_len, m = min(A.chunk_len, np - p0), p = p0 + tid;
    const bool in = tid < m;
    uint32_t k = 0u, t = 0u;
    float4 lo = ident_lo(), hi = ident_hi();
    if (in) {
        k = __ldcg(K + p);
        t = min(__ldcg(V + p), (uint32_t)(A.nt - 1));
        // A triangle whose corners are all NaN on an axis has a NaN box, which holds no point.
        // As a leaf it is empty on that axis, so that the walks test boxes by their gaps;
        // a union takes neither a NaN nor an empty axis in.
        const f4x2 b = ld8_cg(A.tri_box + 2 * t);
        lo = make_float4(fminf(b.a.x, inf), fminf(b.a.y, inf), fminf(b.a.z, inf), 0.0f);
        hi = make_float4(fmaxf(b.b.x, -inf), fmaxf(b.b.y, -inf), fmaxf(b.b.z, -inf), 0.0f);
    }
    // the counts of the chunks before (most are there by the time they are needed)
    uint32_t cw = !BIG && tid < chunk ? ld_volatile(A.ucnt + tid) : CNT_READY;
    S.code[tid + 1] = k;
    if (tid == 0) S.code[0] = p0 > 0 ? __ldcg(K + p0 - 1) : 0u;
    if (warp == 0) S.next[lane] = p0 + m + lane < np ? __ldcg(K + p0 + m + lane) : 0xffffffffu;
    S.flag[tid] = 0u;
    if (lane == 0) S.pbits[warp] = 0u;
    __syncthreads();
    const bool first = in && (BIG || p == 0 || k != S.code[tid]);
    int cnt = m, rank = tid;
    if constexpr (!BIG) {
        const unsigned fb = __ballot_sync(0xffffffffu, first);
        if (lane == 0) S.wcnt[warp] = (uint32_t)__popc(fb);
        __syncthreads();
        const uint32_t wc = lane < RW ? S.wcnt[lane] : 0u;
        cnt = (int)__reduce_add_sync(0xffffffffu, wc);
        rank = (int)__reduce_add_sync(0xffffffffu, lane < warp ? wc : 0u) + __popc(fb & ((1u << lane) - 1u));
        if (tid == 0) st_volatile(A.ucnt + chunk, CNT_READY | (uint32_t)cnt);
    }
    if (first && rank == 0) S.delta[0] = p == 0 ? -1 : __clz((int)(k ^ S.code[tid]));
    const uint32_t* lc = S.code + 1;  // the leaves' codes
    if (!BIG && cnt != m) {           // some position is not a leaf: close the ranks up
        lc = S.lcode;
        if (first) {
            S.lcode[rank] = k;
            S.ltri[rank] = t;
            S.lo[rank][0] = lo;
            S.hi[rank][0] = hi;
        }
        __syncthreads();
        if (tid < cnt) {
            k = S.lcode[tid];
            t = S.ltri[tid];
            lo = S.lo[tid][0];
            hi = S.hi[tid][0];
        }
    }
    f4x2 leaf{};
    if (tid < cnt) leaf = ld8_cg(A.tri_leaf + 2 * t);
    if (tid + 1 < cnt) S.delta[tid + 1] = __clz((int)(k ^ lc[tid + 1]));
    if (warp == 0 && cnt > 0) {  // the boundary to the next leaf, wherever it is
        const uint32_t last = lc[cnt - 1];
        const int e = p0 + m;
        const unsigned b = __ballot_sync(0xffffffffu, e + lane < np && S.next[lane] != last);
        if (lane == 0) {
            int d = -1;
            if (b) {
                d = __clz((int)(last ^ S.next[__ffs(b) - 1]));
            } else if (!BIG && e + 32 < np) {  // more than 32 copies of the code follow: the first larger one
                int l = e + 32, len = np - l;
                while (len > 0) {
                    const int h = len >> 1;
                    if (__ldcg(K + l + h) <= last) {
                        l += h + 1;
                        len -= h + 1;
                    } else {
                        len = h;
                    }
                }
                if (l < np) d = __clz((int)(last ^ __ldcg(K + l)));
            }
            S.delta[cnt] = d;
        }
    }
    __syncthreads();
    int l = tid, r = tid, link = ~tid;  // the current subtree: leaf range, link (local numbers)
    bool live = tid < cnt;              // still climbing
    bool is_root = false, is_a = false;
    int pend = -1, out = -2;  // local node where the climb stopped: one of the chunk's, or one outside it
    int dl = live ? S.delta[l] : 0, dr = live ? S.delta[r + 1] : 0;  // boundaries l - 1 and r
    for (int level = 0; live; ++level) {
        if (level > 64) {  // a climb is at most 31 levels over distinct 30-bit codes
            atomicOr(A.err, ERR_TIMEOUT);
            break;
        }
        if (dl < 0 && dr < 0) {
            is_root = true;
            break;
        }
        is_a = dr > dl;  // the parent extends to the right: this node is child A
        const int g = is_a ? r : l - 1;
        if (g < 0 || g > cnt - 2) {  // split outside the chunk
            out = g;
            break;
        }
        const int side = is_a ? 0 : 1;
        S.lo[g][side] = make_float4(lo.x, lo.y, lo.z, __int_as_float(link));
        S.hi[g][side] = make_float4(hi.x, hi.y, hi.z, __int_as_float(is_a ? far_end(l, dl) : far_end(r, dr)));
        __threadfence_block();
        if (atomicOr(&S.flag[g], 1u << side) == 0u) {  // first to arrive: the sibling may be in another chunk
            pend = g;
            break;
        }
        __threadfence_block();
        // second to arrive: the sibling's side of the slot is complete
        const float4 olo = S.lo[g][side ^ 1], ohi = S.hi[g][side ^ 1];
        const int far = __float_as_int(ohi.w);
        if (is_a) {
            merge_ab(lo, hi, olo, ohi, lo, hi);
            r = far_leaf(far);
            dr = far_delta(far);
        } else {
            merge_ab(olo, ohi, lo, hi, lo, hi);
            l = far_leaf(far);
            dl = far_delta(far);
        }
        link = g;
    }
    int base = p0;  // leaves before the chunk
    if constexpr (!BIG) {
        uint32_t before = 0;
        for (int c = tid; c < chunk; c += RB) {
            int spins = 0;
            if (c != tid) cw = ld_volatile(A.ucnt + c);
            while (!(cw & CNT_READY)) {
                if (++spins > SPIN_LIMIT) {
                    atomicOr(A.err, ERR_TIMEOUT);
                    break;
                }
                __nanosleep(32);
                cw = ld_volatile(A.ucnt + c);
            }
            before += cw & ~CNT_READY;
        }
        before = __reduce_add_sync(0xffffffffu, before);
        if (lane == 0) S.wsum[warp] = before;
        __syncthreads();
        base = (int)__reduce_add_sync(0xffffffffu, lane < RW ? S.wsum[lane] : 0u);
    } else {
        __syncthreads();  // every climb is done
    }
    const auto global_link = [&](float w) {
        const int v = __float_as_int(w);
        return __int_as_float(v >= 0 ? v + base : v - base);
    };
    if (!BIG && tid == 0 && chunk == A.chunks - 1) A.root->n_leaves = base + cnt;
    if (is_root) {  // the whole tree in one chunk; a single leaf has no root node
        A.root->root = l == r ? -1 : link + base;
        A.root->top_lo = make_float4(lo.x, lo.y, lo.z, 0.0f);
        A.root->top_hi = make_float4(hi.x, hi.y, hi.z, 0.0f);
    }
    int up = -2;  // a piece's parent
    if (out != -2) up = out;
    else if (pend >= 0 && S.flag[pend] != 3u) up = pend;
    const bool piece = tid < cnt && up != -2;
    if (piece) atomicOr(&S.pbits[l >> 5], 1u << (l & 31));
    __syncthreads();
    if (piece) {
        int ord = __popc(S.pbits[l >> 5] & ((1u << (l & 31)) - 1u));
        for (int w = 0; w < (l >> 5); ++w) ord += __popc(S.pbits[w]);
        if (ord < MAX_PIECES) {
            S.plo[ord][0] = lo.x; S.plo[ord][1] = lo.y; S.plo[ord][2] = lo.z;
            S.phi[ord][0] = hi.x; S.phi[ord][1] = hi.y; S.phi[ord][2] = hi.z;
            S.pend[ord] = r;
        }
        if (up + base >= 0)  // always, unless a wait for the counts gave up
            write_side(A.nodes, A.range, up + base, is_a, lo, hi, link >= 0 ? link + base : link - base, l + base,
                       r + base);
    }
    __syncthreads();
    if (warp < 2) {  // warp 0 from the left (prefix records), warp 1 from the right (suffix records)
        const bool right = warp == 1;
        int np = lane < RW ? __popc(S.pbits[lane]) : 0;
        np = min((int)__reduce_add_sync(0xffffffffu, np), MAX_PIECES);
        int d[2], j[2], m2 = BIG_DELTA;
        float4 blo[2], bhi[2], lo2 = ident_lo(), hi2 = ident_hi();  // and of the lane's pair
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int e = right ? MAX_PIECES - 1 - (2 * lane + q) : 2 * lane + q;
            const bool ok = e < np;
            j[q] = ok ? S.pend[e] : 0;
            d[q] = ok ? S.delta[j[q] + 1] : BIG_DELTA;
            if (d[q] < 0) d[q] = BIG_DELTA;  // past the last boundary
            blo[q] = ok ? make_float4(S.plo[e][0], S.plo[e][1], S.plo[e][2], 0.0f) : ident_lo();
            bhi[q] = ok ? make_float4(S.phi[e][0], S.phi[e][1], S.phi[e][2], 0.0f) : ident_hi();
            m2 = min(m2, d[q]);
            box_union(lo2, hi2, blo[q], bhi[q]);
        }
        // one copy of the scan's step: this code runs once per chunk, so its length is
        // instruction fetch time (2.4 us for both directions unrolled in one warp)
#pragma unroll 1
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, m2, o);
            const float4 xl = shfl_f4(lo2, o), xh = shfl_f4(hi2, o);
            if (lane >= o) {
                m2 = min(m2, x);
                box_union(lo2, hi2, xl, xh);
            }
        }
        if (lane == 31 && !right) {
            cv.cmin[chunk] = m2;
            st8(cv.cbox + 2 * chunk, lo2, hi2);
        }
        // over the lanes before this one
        int em = __shfl_up_sync(0xffffffffu, m2, 1);
        float4 elo = shfl_f4(lo2, 1), ehi = shfl_f4(hi2, 1);
        if (lane == 0) {
            em = BIG_DELTA;
            elo = ident_lo();
            ehi = ident_hi();
        }
        const bool rec[2] = {d[0] < em, d[1] < min(em, d[0])}, span[2] = {d[0] != BIG_DELTA, d[1] != BIG_DELTA};
        const unsigned lt = (1u << lane) - 1u;
        const unsigned r_0 = __ballot_sync(0xffffffffu, rec[0]), r_1 = __ballot_sync(0xffffffffu, rec[1]);
        const unsigned t_0 = __ballot_sync(0xffffffffu, span[0]), t_1 = __ballot_sync(0xffffffffu, span[1]);
        int ir = __popc(r_0 & lt) + __popc(r_1 & lt), it = __popc(t_0 & lt) + __popc(t_1 & lt);
        int2* const out_rec = (right ? cv.srec : cv.prec) + 32 * chunk;
        float4* const out_box = (right ? cv.sbox : cv.pbox) + 64 * chunk;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            // the chunk's leaves up to the boundary include the piece before it; those after it do not
            float4 ilo = elo, ihi = ehi;
            box_union(ilo, ihi, blo[q], bhi[q]);
            if (rec[q] && ir < 32) {
                out_rec[ir] = make_int2(j[q] + base, d[q]);
                st8(out_box + 2 * ir, right ? elo : ilo, right ? ehi : ihi);
                ++ir;
            }
            if (span[q] && !right) cv.top[MAX_PIECES * chunk + it++] = make_int2(j[q] + base, d[q]);
            elo = ilo;
            ehi = ihi;
        }
        if (lane == 0) {
            cv.rcnt[2 * chunk + (right ? 1 : 0)] =
                (uint32_t)min(__popc(r_0) + __popc(r_1), 32) | (uint32_t)(__popc(t_0) + __popc(t_1)) << 16;
        }
    }
    // meanwhile the other warps write the leaves, and the nodes whose children both arrived here
    if (tid < cnt) {
        st8(A.leaves + 2 * (base + tid), leaf.a, leaf.b);
        if (!BIG) {
            A.ucode[base + tid] = k;
            A.utri[base + tid] = t;
        }
    }
    if (tid < cnt - 1 && S.flag[tid] == 3u) {
        const int g = base + tid;
        const float4 nal = S.lo[tid][0], nah = S.hi[tid][0], nbl = S.lo[tid][1], nbh = S.hi[tid][1];
        st8(&A.nodes[g].a_lo, make_float4(nal.x, nal.y, nal.z, global_link(nal.w)),
            make_float4(nah.x, nah.y, nah.z, 0.0f));
        st8(&A.nodes[g].b_lo, make_float4(nbl.x, nbl.y, nbl.z, global_link(nbl.w)),
            make_float4(nbh.x, nbh.y, nbh.z, 0.0f));
        A.range[g] = make_int2(far_leaf(__float_as_int(nah.w)) + base, far_leaf(__float_as_int(nbh.w)) + base);
    }
    __syncthreads();  // the shared arrays are reused by the CTA's next chunk
}

// First record (in the records' order) of chunk c with delta below d whose position is
// left of g (right of g, with right); g < 0: any position.  -1: none.
__device__ __forceinline__ int first_record(const int2* rec, int count, int g, int d, bool right, int lane,
                                            int2& out) {
    const int2 q = lane < count ? __ldcg(rec + lane) : make_int2(0, BIG_DELTA);
    const bool hit = lane < count && q.y < d && (g < 0 || (right ? q.x > g : q.x < g));
    const unsigned b = __ballot_sync(0xffffffffu, hit);
    if (!b) return -1;
    const int k = __ffs(b) - 1;
    out = make_int2(__shfl_sync(0xffffffffu, q.x, k), __shfl_sync(0xffffffffu, q.y, k));
    return k;
}

// The chunk summaries as the spanning nodes read them: from shared memory (STAGED) or,
// for bodies of more than TOP_STAGED chunks, where they are.  Those bodies have summaries of
// 32 chunks too (phase_groups), or the node at the root alone would read every chunk's, one
// round of 32 after another, and look at their slots 32 at a time (phase_top): 1.3 M triangles
// with distinct codes 219 -> 208 us a rebuild.
template <bool STAGED>
struct Summaries {
    const ChunkView& cv;
    const TopSmem& S;
    __device__ __forceinline__ int min_delta(int c) const { return STAGED ? S.cmin[c] : __ldcg(cv.cmin + c); }
    // records of chunk c from the left / from the right, and its nodes that span chunks
    __device__ __forceinline__ int prefixes(int c) const { return (int)(counts(2 * c) & 0xffffu); }
    __device__ __forceinline__ int suffixes(int c) const { return (int)(counts(2 * c + 1) & 0xffffu); }
    __device__ __forceinline__ int nodes(int c) const { return (int)(counts(2 * c) >> 16); }
    __device__ __forceinline__ uint32_t counts(int i) const { return STAGED ? S.rcnt[i] : __ldcg(cv.rcnt + i); }
    __device__ __forceinline__ void add_box(int c, float4& lo, float4& hi) const {
        if (STAGED)
            box_union(lo, hi, make_float4(S.lo[c][0], S.lo[c][1], S.lo[c][2], 0.0f),
                      make_float4(S.hi[c][0], S.hi[c][1], S.hi[c][2], 0.0f));
        else {
            const f4x2 b = ld8_cg(cv.cbox + 2 * c);
            box_union(lo, hi, b.a, b.b);
        }
    }
    // the leaf boxes of chunks [a, b), over the lanes
    __device__ __forceinline__ void add_boxes(int a, int b, int lane, float4& lo, float4& hi) const {
        const int ga = (a + 31) >> 5, gb = b >> 5;  // whole groups
        const bool grouped = !STAGED && ga < gb;
        for (int e = a + lane; e < (grouped ? 32 * ga : b); e += 32) add_box(e, lo, hi);
        if (grouped) {
            for (int g = ga + lane; g < gb; g += 32) {
                const f4x2 x = ld8_cg(cv.gbox + 2 * g);
                box_union(lo, hi, x.a, x.b);
            }
            if (32 * gb + lane < b) add_box(32 * gb + lane, lo, hi);
        }
    }
    // of the entries v(i), i from `from` in steps of +1 or -1 up to the bounds, the first below d
    template <class Value>
    __device__ __forceinline__ static int first_below(Value v, int from, int n, int d, bool right, int lane) {
        for (int b = from; right ? b < n : b >= 0; b += right ? 32 : -32) {
            const int i = right ? b + lane : b - lane;
            const unsigned h = __ballot_sync(0xffffffffu, i >= 0 && i < n && v(i) < d);
            if (h) return right ? b + __ffs(h) - 1 : b - (__ffs(h) - 1);
        }
        return -1;
    }
    // nearest chunk left of c (right of c) whose min delta is below d; -1: none
    __device__ int nearest(int c, int F, int d, bool right, int lane) const {
        const auto chunk = [&](int i) { return min_delta(i); };
        if (STAGED) return first_below(chunk, right ? c + 1 : c - 1, F, d, right, lane);
        const int g = c >> 5, in = 32 * g + lane;  // the rest of the chunk's own group
        const unsigned h = __ballot_sync(0xffffffffu, (right ? in > c : in < c) && in < F && min_delta(in) < d);
        if (h) return right ? 32 * g + __ffs(h) - 1 : 32 * g + 31 - __clz(h);
        const auto group = [&](int i) { return __ldcg(cv.gmin + i); };
        const int f = first_below(group, right ? g + 1 : g - 1, (F + 31) >> 5, d, right, lane);
        return f < 0 ? -1 : first_below(chunk, right ? 32 * f : min(32 * f + 31, F - 1), F, d, right, lane);
    }
};

// min delta and leaf box union of every 32 chunks, a warp each
__device__ void phase_groups(const RebuildArgs& A, int F) {
    const ChunkView& cv = A.cv;
    const int lane = (int)(threadIdx.x & 31u);
    for (int g = blockIdx.x * RW + (int)(threadIdx.x >> 5); 32 * g < F; g += gridDim.x * RW) {
        const int c = 32 * g + lane;
        int d = BIG_DELTA;
        float4 lo = ident_lo(), hi = ident_hi();
        if (c < F) {
            d = __ldcg(cv.cmin + c);
            const f4x2 b = ld8_cg(cv.cbox + 2 * c);
            box_union(lo, hi, b.a, b.b);
        }
        d = __reduce_min_sync(0xffffffffu, d);
        warp_box_reduce(lo, hi);
        if (lane == 0) {
            cv.gmin[g] = d;
            st8(cv.gbox + 2 * g, lo, hi);
        }
    }
}

// One node that spans chunks, by one warp: the range ends are the nearest boundaries
// with a smaller delta on either side (the first suffix / prefix record past the node
// with a smaller delta, in the node's chunk or in the nearest chunk with a smaller min),
// the box is the union of the leaf boxes in the range (the records' partial unions and
// whole chunks between), and the node enters its parent (the range end with the larger
// delta) as the climb would have put it there.
template <bool STAGED>
__device__ void top_node(const RebuildArgs& A, const Summaries<STAGED>& sum, int c, int sl, int n, int F, int lane) {
    const ChunkView& cv = A.cv;
    const int2 item = __ldcg(cv.top + MAX_PIECES * c + sl);
    const int g = item.x, d = item.y;
    if (g < 0 || g > n - 2) {
        if (lane == 0) atomicOr(A.err, ERR_TIMEOUT);
        return;
    }
    // both sides' searches first, then the loads they lead to
    int2 ql, qr;
    int kl = first_record(cv.srec + 32 * c, sum.suffixes(c), g, d, false, lane, ql), cl = c;
    int kr = first_record(cv.prec + 32 * c, sum.prefixes(c), g, d, true, lane, qr), cr = c;
    if (kl < 0) {
        cl = sum.nearest(c, F, d, false, lane);
        if (cl >= 0) kl = first_record(cv.srec + 32 * cl, sum.suffixes(cl), -1, d, false, lane, ql);
    }
    if (kr < 0) {
        cr = sum.nearest(c, F, d, true, lane);
        if (cr >= 0) kr = first_record(cv.prec + 32 * cr, sum.prefixes(cr), -1, d, true, lane, qr);
    }
    int jl = -1, dlft = -1, jr = n - 1, drgt = -1;  // leaves jl + 1 .. jr
    float4 lo = ident_lo(), hi = ident_hi();
    if (kl >= 0) {
        jl = ql.x;
        dlft = ql.y;
        const f4x2 b = ld8_cg(cv.sbox + 2 * (32 * cl + kl));
        box_union(lo, hi, b.a, b.b);
    } else {
        cl = -1;
    }
    if (kr >= 0) {
        jr = qr.x;
        drgt = qr.y;
        const f4x2 b = ld8_cg(cv.pbox + 2 * (32 * cr + kr));
        box_union(lo, hi, b.a, b.b);
    } else {
        cr = F;
    }
    float4 ul = ident_lo(), uh = ident_hi();
    sum.add_boxes(cl + 1, cr, lane, ul, uh);
    warp_box_reduce(ul, uh);
    box_union(lo, hi, ul, uh);
    if (lane == 0) {
        if (jl < 0 && jr == n - 1) {
            A.root->root = g;
            A.root->top_lo = lo;
            A.root->top_hi = hi;
        } else {
            const bool is_a = drgt > dlft;
            write_side(A.nodes, A.range, is_a ? jr : jl, is_a, lo, hi, g, jl + 1, jr);
        }
    }
}

// The nodes whose leaf range spans chunks, one warp each, independently.  Each CTA stages
// the summaries it searches (28 bytes a chunk) and the running count of the chunks' nodes,
// by which the warps share the nodes out.
template <bool BIG>
__device__ void phase_top(const RebuildArgs& A, int F, TopSmem& S, uint32_t* s_scan) {
    const ChunkView& cv = A.cv;
    const int lane = (int)(threadIdx.x & 31u);
    const int n = __ldcg(&A.root->n_leaves);
    const uint32_t w0 = blockIdx.x * RW + (threadIdx.x >> 5), nw = gridDim.x * RW;
    if (BIG && F > TOP_STAGED) {  // slot s of every chunk before slot s + 1 of any: the low ones are occupied
        const Summaries<false> sum{cv, S};
        for (uint64_t it = w0; it < (uint64_t)F * MAX_PIECES; it += 32ull * nw) {  // a warp's next 32 slots
            const uint64_t my = it + (uint64_t)lane * nw;
            const int c = (int)(my % (uint32_t)F), sl = (int)(my / (uint32_t)F);
            unsigned used = __ballot_sync(0xffffffffu, sl < MAX_PIECES && sl < sum.nodes(c));
            for (; used; used &= used - 1u) {
                const int from = __ffs(used) - 1;
                top_node<false>(A, sum, __shfl_sync(0xffffffffu, c, from), __shfl_sync(0xffffffffu, sl, from), n, F, lane);
            }
        }
        return;
    }
    const int i = 2 * (int)threadIdx.x;
    const uint2 r0 = i < F ? __ldcg(reinterpret_cast<const uint2*>(cv.rcnt) + i) : make_uint2(0u, 0u);
    const uint2 r1 = i + 1 < F ? __ldcg(reinterpret_cast<const uint2*>(cv.rcnt) + i + 1) : make_uint2(0u, 0u);
    const uint32_t c0 = r0.x >> 16, c1 = r1.x >> 16;
    reinterpret_cast<uint2*>(S.rcnt)[i] = r0;
    reinterpret_cast<uint2*>(S.rcnt)[i + 1] = r1;
    for (int c = threadIdx.x; c < F; c += RB) {
        const f4x2 b = ld8_cg(cv.cbox + 2 * c);
        S.cmin[c] = __ldcg(cv.cmin + c);
        S.lo[c][0] = b.a.x; S.lo[c][1] = b.a.y; S.lo[c][2] = b.a.z;
        S.hi[c][0] = b.b.x; S.hi[c][1] = b.b.y; S.hi[c][2] = b.b.z;
    }
    const uint32_t incl = block_scan_incl(c0 + c1, s_scan);
    S.pre[i] = incl - c0 - c1;
    S.pre[i + 1] = incl - c1;
    if (i == TOP_STAGED - 2) S.pre[TOP_STAGED] = incl;
    __syncthreads();
    const Summaries<true> sum{cv, S};
    const uint32_t total = S.pre[TOP_STAGED];
    for (uint32_t it = w0; it < total; it += nw) {
        int lo = 0, hi = F;  // the chunk: S.pre[lo] <= it < S.pre[hi]
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (S.pre[mid] <= it) lo = mid;
            else hi = mid;
        }
        top_node<true>(A, sum, lo, (int)(it - S.pre[lo]), n, F, lane);
    }
}

// ---- the launch -----------------------------------------------------------------------------------
// BIG: more triangles than TOP_STAGED chunks hold.  An instance of its own, so that the
// others' code stays as short as it is (with both in one, 327,680 triangles took 72 -> 78 us).
template <bool BIG>
__global__ void __launch_bounds__(RB, 2) k_rebuild(const RebuildArgs A) {
    extern __shared__ __align__(16) unsigned char rb_smem[];
    __shared__ uint32_t s_scan[32];
    __shared__ float s_red[6 * RW];
    __shared__ float s_frame[8];
    __shared__ int s_ok, s_claim;
    uint32_t target = 0;
    const int nt = A.nt;
    // the last build's sorted list (keys[cur], vals[cur]) and codes are usable: read
    // before any CTA can change the root record
    const bool coherent = A.coherent && ld_volatile(reinterpret_cast<const uint32_t*>(&A.root->perm_valid)) != 0u;
    const int cur = coherent ? (int)ld_volatile(reinterpret_cast<const uint32_t*>(&A.root->sorted)) & 1 : 1;
    // what the later phases need at zero (read only after the next barrier)
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        A.chg[0] = 0u;
        A.root->n_tris = nt;
        A.root->nodes = A.nodes;
        A.root->leaves = A.leaves;
    }
    {
        const int k0 = blockIdx.x * RB + threadIdx.x, step = gridDim.x * RB;
        const size_t zw = (size_t)PASSES * RADIX + (size_t)PASSES * A.tiles_sort * RADIX + PASSES;
        for (size_t k = k0; k < zw; k += step) A.ghist[k] = 0u;
        for (int k = k0; k < BK_MAX; k += step) A.bcnt[k] = 0u;
        for (int k = k0; k < A.chunks; k += step) A.ucnt[k] = 0u;
    }
    phase_verts(A);
    bool ok = true;
    f3 cen[BOX_BATCH];
    uint32_t old[BOX_BATCH];  // the last build's codes of the same triangles
#pragma unroll
    for (int q = 0; q < BOX_BATCH; ++q) {
        const int t = (blockIdx.x + q * gridDim.x) * RB + threadIdx.x;
        cen[q] = mk3(0.0f, 0.0f, 0.0f);
        old[q] = coherent && t < nt ? A.codes[t] : 0u;
    }
    if (!BIG && A.direct) {
        phase_boxes<true>(A, s_red, cen);
    } else {
        ok = grid_barrier(A.sync, target, ok, A.err, &s_ok);
        if (ok) phase_boxes<false>(A, s_red, cen);
    }
    ok = grid_barrier(A.sync, target, ok, A.err, &s_ok);
    if (ok) phase_codes(A, coherent, s_red, s_frame, cen, old);
    ok = grid_barrier(A.sync, target, ok, A.err, &s_ok);
    // the sort: same decision in every CTA (from words complete at the barrier)
    const uint32_t nchg = ld_volatile(A.chg);
    int after = cur;  // buffer holding this build's sorted list
    if (coherent && nchg <= (uint32_t)CHG_CAP) {
        if (nchg > 0u) {  // else every code is as before: the last build's list stands
            after = cur ^ 1;
            if (ok)
                phase_merge(A, (int)nchg, A.keys[cur], A.vals[cur], A.keys[after], A.vals[after],
                            *reinterpret_cast<MergeSmem*>(rb_smem));
            ok = grid_barrier(A.sync, target, ok, A.err, &s_ok);
        }
    } else {
        bool sorted = false;
        if (!BIG && (coherent ? A.buckets > 0 : nt <= SAMPLED_MAX)) {
            BucketSmem& S = *reinterpret_cast<BucketSmem*>(rb_smem);
            const int nb = A.buckets;
            after = cur ^ 1;
            if (!coherent && nb > 1) {
                if (ok) phase_sample(A, nb * OVERSAMPLE, S);
                ok = grid_barrier(A.sync, target, ok, A.err, &s_ok);
            }
            if (ok) phase_scatter(A, nb, coherent ? A.keys[cur] : nullptr, A.vals[cur], S);
            ok = grid_barrier(A.sync, target, ok, A.err, &s_ok);
            sorted = buckets_fit(A, nb, S, s_scan);
            if (sorted) {
                if (ok) phase_bucket_sort(A, nb, A.keys[after], A.vals[after], S);
                ok = grid_barrier(A.sync, target, ok, A.err, &s_ok);
            }
        }
        if (!sorted) {
            if (ok) phase_hist(A, reinterpret_cast<uint32_t*>(rb_smem));
            ok = grid_barrier(A.sync, target, ok, A.err, &s_ok);
            for (int p = 0; p < PASSES; ++p) {
                if (ok) phase_sort_pass(A, p, *reinterpret_cast<SortSmem*>(rb_smem), s_scan, &s_claim);
                ok = grid_barrier(A.sync, target, ok, A.err, &s_ok);
            }
            after = (PASSES - 1) & 1;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        // the sort buffers now hold this build's list, unless some wait gave up
        const bool bad = !ok || (ld_volatile(reinterpret_cast<const uint32_t*>(A.err)) & ERR_TIMEOUT) != 0u;
        A.root->perm_valid = bad ? 0 : 1;
        A.root->sorted = after;
    }
    const uint32_t *K = A.keys[after], *V = A.vals[after];
    int np = nt, F = A.chunks;  // positions the build goes through, and their chunks
    if constexpr (BIG) {
        if (ok) phase_unique_count(A, K, s_scan);
        ok = grid_barrier(A.sync, target, ok, A.err, &s_ok);
        if (ok) np = phase_unique_write(A, K, V, s_scan);
        ok = grid_barrier(A.sync, target, ok, A.err, &s_ok);
        K = A.ucode;
        V = A.utri;
        F = (np + A.chunk_len - 1) / A.chunk_len;
    }
    if (ok)
        for (int c = blockIdx.x; c < F; c += gridDim.x)
            build_chunk<BIG>(A, c, np, K, V, *reinterpret_cast<BuildSmem*>(rb_smem));
    ok = grid_barrier(A.sync, target, ok, A.err, &s_ok);
    if (BIG && F > TOP_STAGED) {
        if (ok) phase_groups(A, F);
        ok = grid_barrier(A.sync, target, ok, A.err, &s_ok);
    }
    if (ok) phase_top<BIG>(A, F, *reinterpret_cast<TopSmem*>(rb_smem), s_scan);
    // the last CTA out leaves both counters at zero for the next launch
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(A.sync + 1, 1u) == gridDim.x - 1u) {
            atomicExch(A.sync, 0u);
            atomicExch(A.sync + 1, 0u);
        }
    }
}

// Self-test of the grid barrier's bounded wait: one CTA waits for an arrival count
// that no other CTA will bring; the wait gives up after kGridWaitNs, records
// ERR_TIMEOUT and returns.
__global__ void k_selftest_grid_wait(uint32_t* ctr, int* err) {
    __shared__ int s_ok;
    uint32_t target = 1;  // as if one barrier of this one-CTA launch had passed
    (void)grid_barrier(ctr, target, true, err, &s_ok);
}

// Self-test of the look-back's bounded wait: one thread looks back from tile 1 at a
// status word (tile 0's) that nothing publishes; the walk gives up after SPIN_LIMIT
// sleeps, records ERR_TIMEOUT and returns.
__global__ void k_selftest_look_back(const uint32_t* status, int* err) {
    if (threadIdx.x == 0) (void)look_back(status, 1, 1, err);
}

inline int cdiv(int a, int b) { return (a + b - 1) / b; }

// CTAs of k_rebuild that fit on the device at once (cooperative launch limit)
template <bool BIG>
int resident_ctas() {
    static std::mutex mu;
    static int cached[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    std::lock_guard<std::mutex> lk(mu);
    if (!cached[dev]) {
        int sms = 0, per = 0;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_rebuild<BIG>, RB, kSmemBytes) != cudaSuccess) return 0;
        cached[dev] = sms * per;
    }
    return cached[dev];
}

// Positions per chunk of the build.  Two CTAs an SM take the chunks in turn, so the chunks of
// the rounds that RB positions would need are made equal: 327,680 triangles are 640 chunks
// of 512, two rounds and 32 chunks more, or 854 of 384 (rebuild 75.7 -> 72.2 us; of 256, 88.5:
// four rounds).  A small body's are no shorter than 256 (19,584 triangles: 512 22.2 us, 256
// 20.9, 128 22.7, its spanning nodes take what the build gains), and a body whose summaries
// would no longer fit the spanning-node phase's shared memory for it keeps them there.
int chunk_length(int nt) {
    constexpr int kResident = 2 * SPREAD_CTAS, kLeast = 256;
    const int rounds = cdiv(cdiv(nt, RB), kResident);
    int len = std::max(cdiv(nt, rounds * kResident), kLeast);
    if (nt <= TOP_STAGED * RB) len = std::max(len, cdiv(nt, TOP_STAGED));
    return std::min(RB, (len + 31) / 32 * 32);
}

}  // namespace

void BvhBuffers::plan(Arena& a, int nv_, int nt_, bool normals, bool walked) {
    nv = nv_;
    nt = nt_;
    has_normals = normals;
    tiles_sort = nt > 0 ? cdiv(nt, SORT_TILE) : 0;
    chunk_len = chunk_length(std::max(nt, 1));
    chunks = cdiv(std::max(nt, 1), chunk_len);
    // a chunk per CTA at most, but for a small body enough CTAs that the phases before
    // the build spread over the SMs
    max_ctas = std::max(chunks, std::min(SPREAD_CTAS, cdiv(std::max(nt, 1), RB / 4)));
    int ni = nt > 1 ? nt - 1 : 1;
    a.want(&xyz_in, (size_t)nv * 3 + 4);
    a.want(&nrm_in, (size_t)nv * 3 + 4);
    a.want(&verts, (size_t)nv + 1);
    a.want(&tris, (size_t)nt * 3 + 4);
    a.want(&tri_box, (size_t)nt * 2 + 2);
    a.want(&tri_leaf, (size_t)nt * 2 + 2);
    a.want(&codes, (size_t)nt + 1);
    for (int k = 0; k < 2; ++k) {
        a.want(&keys[k], (size_t)nt + 1);
        a.want(&vals[k], (size_t)nt + 1);
    }
    a.want(&ucode, (size_t)nt + 1);
    a.want(&utri, (size_t)nt + 1);
    a.want(&nodes, (size_t)ni);
    a.want(&leaves, (size_t)nt * 2 + 2);
    a.want(&range, (size_t)ni);
    a.want(&cmin, (size_t)chunks);
    a.want(&cbox, 2 * (size_t)chunks);
    a.want(&srec, 32 * (size_t)chunks);
    a.want(&sbox, 64 * (size_t)chunks);
    a.want(&prec, 32 * (size_t)chunks);
    a.want(&pbox, 64 * (size_t)chunks);
    a.want(&rcnt, 2 * (size_t)chunks);
    a.want(&top, (size_t)MAX_PIECES * chunks);
    if (chunks > TOP_STAGED) {
        a.want(&gmin, (size_t)cdiv(chunks, 32));
        a.want(&gbox, 2 * (size_t)cdiv(chunks, 32));
    }
    if (!walked) a.want(&root, 1);
    // histograms | sort status (PASSES x tiles x RADIX) | sort counters (the launch
    // clears them) | bucket counts | CTA box unions | chunk leaf counts | change list | barrier counters
    scratch_words = (size_t)PASSES * RADIX + (size_t)PASSES * tiles_sort * RADIX + PASSES;
    a.want(&scratch, scratch_words);
    a.want(&bcnt, (size_t)BK_MAX);
    a.want(&bkey, (size_t)SAMPLES);
    buckets = nt <= BK_MAX * (BK_CAP / 2) ? std::min(cdiv(std::max(nt, 1), BK_TARGET), BK_MAX) : 0;
    if (walked) a.want(&bslot, (size_t)buckets * BK_CAP);
    a.want(&part, 8 * (size_t)max_ctas);
    a.want(&ucnt, (size_t)chunks);
    a.want(&chg, 1 + 3 * (size_t)CHG_CAP);
    a.want(&sync, 2);
}

cudaError_t lbvh_build(BvhBuffers& b, float thickness, float box_depth, int* d_err, cudaStream_t s, const float* xyz,
                       const float* nrm, float4* margin_state, int64_t m0, int64_t m1) {
    if (b.nt == 0) return cudaSuccess;
    const bool big = b.chunks > TOP_STAGED;
    const int res = big ? resident_ctas<true>() : resident_ctas<false>();
    if (res <= 0) return cudaErrorLaunchOutOfResources;
    RebuildArgs A;
    A.xyz = xyz ? xyz : b.xyz_in;
    A.nrm = b.has_normals ? (xyz ? nrm : b.nrm_in) : nullptr;
    A.margin_state = margin_state;
    A.m0 = m0;
    A.m1 = m1;
    A.tris = b.tris;
    A.nv = b.nv;
    A.nt = b.nt;
    A.thickness = thickness;
    A.depth = box_depth;
    A.coherent = b.coherent ? 1 : 0;
    A.direct = b.nt <= DIRECT_MAX ? 1 : 0;
    A.tiles_sort = b.tiles_sort;
    A.verts = b.verts;
    A.tri_box = b.tri_box;
    A.tri_leaf = b.tri_leaf;
    A.codes = b.codes;
    for (int k = 0; k < 2; ++k) {
        A.keys[k] = b.keys[k];
        A.vals[k] = b.vals[k];
    }
    A.ucode = b.ucode;
    A.utri = b.utri;
    A.nodes = b.nodes;
    A.leaves = b.leaves;
    A.range = b.range;
    A.root = b.root;
    A.cv = ChunkView{b.cmin, b.cbox, b.srec, b.sbox, b.prec, b.pbox, b.rcnt, b.top, b.gmin, b.gbox};
    A.ghist = b.scratch;
    A.sstat = A.ghist + PASSES * RADIX;
    A.scount = A.sstat + (size_t)PASSES * b.tiles_sort * RADIX;
    A.part = b.part;
    A.ucnt = b.ucnt;
    A.chg = b.chg;
    A.sync = b.sync;
    A.bcnt = b.bcnt;
    A.bkey = b.bkey;
    // a tree that nobody walks keeps the slots in its node array, which the build writes later
    A.bslot = b.bslot ? b.bslot : reinterpret_cast<unsigned long long*>(b.nodes);
    A.buckets = b.buckets;
    A.chunks = b.chunks;
    A.chunk_len = b.chunk_len;
    A.err = d_err;
    const int grid = std::min(res, b.max_ctas);
    void* args[] = {&A};
    return cudaLaunchCooperativeKernel(big ? (const void*)k_rebuild<true> : (const void*)k_rebuild<false>, dim3(grid),
                                       dim3(RB), args, kSmemBytes, s);
}

cudaError_t launch_selftest_look_back(const uint32_t* zero_status, int* err, cudaStream_t s) {
    k_selftest_look_back<<<1, 32, 0, s>>>(zero_status, err);
    return cudaGetLastError();
}

cudaError_t launch_selftest_grid_wait(uint32_t* zero_counter, int* err, cudaStream_t s) {
    k_selftest_grid_wait<<<1, 32, 0, s>>>(zero_counter, err);
    return cudaGetLastError();
}

}  // namespace visg
