// visg_lbvh_static.cu — the body LBVH build without any device allocation.
//
// Some callers of this library cannot call cudaMalloc: a host application whose
// own allocator owns the whole device (a pooling allocator or an arena sized at
// start-up), code that runs where allocation is forbidden or would synchronise the
// device at a bad moment, or a plugin that must not change the process's memory
// footprint after initialisation.  visg_lbvh_build_noalloc serves them: the caller
// passes the body (device pointers) and the output arrays, and every temporary the
// build needs (boxes, Morton codes, radix-sort buffers, look-back status words,
// chunk summaries) lives in one file-scope __device__ array, so the call itself
// allocates nothing.
//
// Costs and limits:
//   * the array (VISG_NOALLOC_SCRATCH_BYTES) is reserved on every GPU that loads
//     this library and held until the process exits;
//   * bodies are limited to VISG_NOALLOC_MAX_VERTICES vertices and
//     VISG_NOALLOC_MAX_TRIS triangles; larger inputs are rejected;
//   * all calls share the array and it keeps the last call's contents: the build
//     clears what must start at zero itself, and two calls whose GPU work overlaps
//     (different streams, or different host threads) race on it.
#include <cuda_runtime.h>

#include <mutex>

#include "visg_internal.cuh"

using namespace visg;

namespace {

constexpr size_t kScratchBytes = VISG_NOALLOC_SCRATCH_BYTES;
constexpr int kMaxDevices = 64;

static __device__ __align__(256) unsigned char g_lbvh_scratch[kScratchBytes];

std::mutex g_mu;
void* g_scratch_addr[kMaxDevices] = {};  // device address of g_lbvh_scratch, per device

int bad(int code) { return code; }

// The array's name in host code is a host-side stand-in, not a device address:
// look the address up once per device, with that device current.
int scratch_address(void** out) {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices)
        return bad(VISG_ERR_NO_DEVICE);
    std::lock_guard<std::mutex> lk(g_mu);
    if (!g_scratch_addr[dev]) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_lbvh_scratch);
        if (e != cudaSuccess || !p) return bad(VISG_ERR_CUDA);
        g_scratch_addr[dev] = p;
    }
    *out = g_scratch_addr[dev];
    return VISG_OK;
}

// Reference layout of the links (BRTreeNode, cudaBRT.h:34-115): the root is
// internal node 0; an internal node that is child A takes the index of its last
// leaf, child B of its first; links are +(i+1) internal, -(i+1) leaf.  The node split
// at g over the leaves [l, r] has children over [l, g] and [g + 1, r], so their indices
// are g and g + 1, and it is child A itself when its right end has the longer common
// prefix: each node's links follow from its own range and four codes, in one pass.
// The leaf count goes to the caller from the same launch; -1 if a bounded wait of the
// build gave up or an index was out of range (a triangle's vertex index, or a range
// read from the tree).  The pass runs only on a build that reported no error, and checks
// the range it read before using it: a build whose bounded wait gave up can leave the
// shared array with another call's nodes, and nothing read from there may send a store
// outside the caller's arrays.
// err: [0] the build's error word, [1] blocks of this launch that are done.
__global__ void k_karras(const int2* __restrict__ range, const uint32_t* __restrict__ codes,
                         const BvhRoot* __restrict__ root, int32_t* __restrict__ child_a,
                         int32_t* __restrict__ child_b, int n_tris, int* err, int32_t* n_leaves) {
    const int n = root->n_leaves;
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (*reinterpret_cast<volatile int*>(err) == 0 && n >= 2 && n <= n_tris && g < n - 1) {
        const int2 q = range[g];
        int k = -1;
        if (q.x >= 0 && q.x <= g && q.y > g && q.y < n) {
            const int dl = q.x > 0 ? __clz((int)(codes[q.x - 1] ^ codes[q.x])) : -1;
            const int dr = q.y < n - 1 ? __clz((int)(codes[q.y] ^ codes[q.y + 1])) : -1;
            k = q.x == 0 && q.y == n - 1 ? 0 : dr > dl ? q.y : q.x;
        }
        if (k < 0 || k > n - 2) {
            atomicOr(err, ERR_INDEX);
        } else {
            child_a[k] = q.x == g ? -(g + 1) : g + 1;
            child_b[k] = q.y == g + 1 ? -(g + 2) : g + 2;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(err + 1, 1) == (int)gridDim.x - 1)
            *n_leaves = atomicAdd(err, 0) ? -1 : n;
    }
}

}  // namespace

extern "C" int visg_lbvh_build_noalloc(const float* d_xyz, const float* d_normals, int32_t n_vertices,
                                       const uint32_t* d_tris, int32_t n_tris, float thickness, float box_depth,
                                       uint32_t* d_sorted_codes, int32_t* d_sorted_tris, int32_t* d_child_a,
                                       int32_t* d_child_b, int32_t* d_n_leaves, void* cuda_stream) {
    if (!d_xyz || !d_tris || !d_sorted_codes || !d_sorted_tris || !d_n_leaves || (n_tris > 1 && (!d_child_a || !d_child_b)))
        return bad(VISG_ERR_INVALID_ARG);  // a NULL pointer
    if (n_vertices < 1 || n_tris < 1) return bad(VISG_ERR_INVALID_ARG);  // empty body
    // larger than the static scratch holds: such bodies go through visg_create / visg_update_body
    if (n_vertices > VISG_NOALLOC_MAX_VERTICES || n_tris > VISG_NOALLOC_MAX_TRIS) return bad(VISG_ERR_INVALID_ARG);
    void* base = nullptr;
    if (int r = scratch_address(&base)) return r;
    cudaStream_t s = (cudaStream_t)cuda_stream;

    // carve the build's buffers out of the static array (the same plan the
    // allocating path uses), then point inputs and outputs at the caller's arrays
    BvhBuffers b;
    Arena plan;
    b.plan(plan, n_vertices, n_tris, d_normals != nullptr, false);
    int* d_err = nullptr;
    plan.want(&d_err, 4);
    size_t used = 0;
    for (auto& pl : plan.plan) used += pl.second;
    if (used > kScratchBytes) return bad(VISG_ERR_UNSUPPORTED);  // cannot happen within the size limits
    char* p = (char*)base;
    for (auto& pl : plan.plan) {
        *pl.first = p;
        p += pl.second;
    }
    b.xyz_in = const_cast<float*>(d_xyz);
    b.nrm_in = const_cast<float*>(d_normals);
    b.tris = const_cast<uint32_t*>(d_tris);
    b.ucode = d_sorted_codes;
    b.utri = reinterpret_cast<uint32_t*>(d_sorted_tris);

    // what must start at zero: the build's grid-barrier counters and the error word, which
    // the plan lays side by side at its end (the array holds the last call's data, laid
    // out for its sizes); the build clears its histograms, look-back status words and
    // counters itself
    cudaError_t e = cudaMemsetAsync(b.sync, 0, (size_t)((char*)(d_err + 2) - (char*)b.sync), s);
    if (e == cudaSuccess) e = lbvh_build(b, thickness, box_depth, d_err, s);
    if (e == cudaSuccess) {
        k_karras<<<(unsigned)((n_tris + 255) / 256), 256, 0, s>>>(b.range, b.ucode, b.root, d_child_a, d_child_b,
                                                                  n_tris, d_err, d_n_leaves);
        e = cudaGetLastError();
    }
    return e == cudaSuccess ? VISG_OK : bad(VISG_ERR_CUDA);
}
