// CWBVH build on the GPU, for scenes that change or arrive in batches: the
// same node and triangle layouts as the host builder (cwbvh_build.cpp; the
// layouts the reference traversal decodes, traverse_cwbvh.cuh:77-209), built
// without leaving the device.
//
//   1. compact the TRIANGULO primitives in input order (their index is the
//      prim id, as tinybvh_wrapper.cpp:36-44 numbers them), FP32 vertices;
//   2. 30-bit Morton codes of the triangle centroids, radix-sorted;
//   3. binary radix tree over the sorted codes (Karras 2012, "Maximizing
//      Parallelism in the Construction of BVHs, Octrees, and k-d Trees"),
//      duplicate codes ordered by index;
//   4. boxes, triangle counts and collapse plans bottom-up, one thread per
//      leaf climbing while it is the second child to finish;
//   5. one kernel per wide level, eight lanes per wide node: the lanes expand
//      the node's collapse plan into its up to 8 children (a subtree of <= 3
//      triangles becomes a leaf slot), assign octant slots greedily, quantise
//      the child boxes to 8 bits and reserve contiguous blocks for the inner
//      children and leaf triangles with atomics;
//   6. the reference transform triangles and the watertight triangles in
//      leaf order.
// The tree is a Morton-order (LBVH) tree: it builds in under a millisecond
// for 10^5 triangles, and traverses slower than the host builder's binned-SAH
// tree.
//
// A build is a chain of short dependent kernels, so what counts is the host
// work around them and each kernel's latency: all scratch is one block of a
// bounded stream-ordered pool (cudaMalloc and cudaFree take ~0.3 ms each here:
// the former 25 pairs took most of an 81,920-triangle build),
// the result is one allocation made while the GPU works, the initial values
// come from a kernel, and the levels run in batches whose sizes stay on the
// device (one host read per eight levels instead of one per level).
#include <cuda_runtime.h>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>
#include <thrust/iterator/transform_iterator.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <string>

#include "../../include/tfg_pt.h"
#include "tfg_errors.h"
#include "tfg_runtime.h"

namespace tfg {
namespace {

constexpr int kMaxLeaf = 3;   // the 3-bit unary meta count limits a leaf to 3 triangles

// Box and triangle count of a binary node (or of a triangle), read and
// written as two 16-byte halves.
struct __align__(16) BNode {
    float lo[3];
    int count;
    float hi[3];
    float pad;
};

// Collapse plan of an interior binary node, as in the host builder
// (cwbvh_build.cpp): for a budget of i = 1..8 slots of the wide parent, the
// least SAH cost of the node's subtree and how it is reached (leaf of <= 3
// triangles, a wide node of its own, as with one slot less, or split with k
// slots to the left).  A single triangle has no stored plan: every budget
// costs its leaf.
struct __align__(16) Plan2 {
    float cost[8];
    uint8_t how[8];
    uint8_t split8;       // as a wide node: slots given to the left child
    uint8_t pad[7];
};
static_assert(sizeof(BNode) == 32 && sizeof(Plan2) == 48, "vector loads");
constexpr uint8_t kLeaf = 0, kInternal = 1, kSame = 2, kSplit = 16;
constexpr float kCostWideNode = 1.0f, kCostWideTri = 0.3f;

__device__ __forceinline__ float box_area(const BNode& b) {
    const float dx = fmaxf(b.hi[0] - b.lo[0], 0.0f), dy = fmaxf(b.hi[1] - b.lo[1], 0.0f),
                dz = fmaxf(b.hi[2] - b.lo[2], 0.0f);
    return 2.0f * (dx * dy + dx * dz + dy * dz);
}

__device__ __forceinline__ uint32_t expand_bits(uint32_t v) {   // 10 bits -> every third bit
    v = (v * 0x00010001u) & 0xFF0000FFu;
    v = (v * 0x00000101u) & 0x0F00F00Fu;
    v = (v * 0x00000011u) & 0xC30C30C3u;
    v = (v * 0x00000005u) & 0x49249249u;
    return v;
}

struct IsTriangle {
    __host__ __device__ uint32_t operator()(const TfgPrimitiva& p) const { return p.tipo == TFG_TRIANGULO ? 1u : 0u; }
};

// Order-preserving float <-> uint mapping for atomic min / max.
__device__ __forceinline__ uint32_t fkey(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float funkey(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
}

// Device words of one build.
struct BuildWords {
    uint32_t cb[6];             // centroid bounds as ordered keys: lo.xyz, hi.xyz
    uint32_t next_node, next_tri;
    uint32_t level[66];         // wide nodes of each level
};

// Initial values: empty centroid bounds, the root as the only node of level
// 0 (binary node 0; with one triangle, its leaf), nothing arrived.
__global__ void k_build_init(BuildWords* w, int2* q0, uint32_t* arrivals, uint32_t nt) {
    const uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x;
    for (uint32_t i = i0; i < nt; i += gridDim.x * blockDim.x) arrivals[i] = 0u;
    if (i0 < 6) w->cb[i0] = i0 < 3 ? 0xFFFFFFFFu : 0u;
    if (i0 == 6) w->next_node = 1u;
    if (i0 == 7) w->next_tri = 0u;
    if (i0 >= 8 && i0 < 8 + 66) w->level[i0 - 8] = i0 == 8 ? 1u : 0u;
    if (i0 == 74) *q0 = make_int2(0, 0);
}

// Compacted triangles' FP32 vertices and boxes, and the centroid bounds.
// `pos` counts the triangles up to and including each primitive.
__global__ void __launch_bounds__(256) k_compact(const TfgPrimitiva* __restrict__ p, int n,
                                                 const uint32_t* __restrict__ pos, float* __restrict__ verts,
                                                 BNode* __restrict__ box, BuildWords* words) {
    float clo[3] = {INFINITY, INFINITY, INFINITY}, chi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (p[i].tipo != TFG_TRIANGULO) continue;
        const uint32_t k = pos[i] - 1u;
        const auto& t = p[i].u.triangulo;
        const TfgVec3d* v[3] = {&t.v0, &t.v1, &t.v2};
        BNode b;
        for (int a = 0; a < 3; ++a) { b.lo[a] = INFINITY; b.hi[a] = -INFINITY; }
        for (int c = 0; c < 3; ++c) {
            const float x[3] = {(float)v[c]->x, (float)v[c]->y, (float)v[c]->z};
            for (int a = 0; a < 3; ++a) {
                verts[9 * (size_t)k + 3 * c + a] = x[a];
                b.lo[a] = fminf(b.lo[a], x[a]);
                b.hi[a] = fmaxf(b.hi[a], x[a]);
            }
        }
        b.count = 1;
        b.pad = 0.0f;
        box[k] = b;
        for (int a = 0; a < 3; ++a) {
            const float c = 0.5f * (b.lo[a] + b.hi[a]);
            clo[a] = fminf(clo[a], c);
            chi[a] = fmaxf(chi[a], c);
        }
    }
    __shared__ uint32_t s_cb[6];
    if (threadIdx.x < 6) s_cb[threadIdx.x] = threadIdx.x < 3 ? 0xFFFFFFFFu : 0u;
    __syncthreads();
    for (int a = 0; a < 3; ++a) {
        const uint32_t lo = __reduce_min_sync(0xFFFFFFFFu, fkey(clo[a])), hi = __reduce_max_sync(0xFFFFFFFFu, fkey(chi[a]));
        if ((threadIdx.x & 31) == 0) { atomicMin(&s_cb[a], lo); atomicMax(&s_cb[3 + a], hi); }
    }
    __syncthreads();
    if (threadIdx.x < 3) atomicMin(&words->cb[threadIdx.x], s_cb[threadIdx.x]);
    else if (threadIdx.x < 6) atomicMax(&words->cb[threadIdx.x], s_cb[threadIdx.x]);
}

// The TRIANGULO primitives, compacted.  A warp copies the 200-byte structs of
// its 32 primitives together, 8 bytes per lane and step (a struct per lane
// moves them at a 200-byte stride).
__global__ void __launch_bounds__(256) k_copy_prims(const TfgPrimitiva* __restrict__ p, int n,
                                                    const uint32_t* __restrict__ pos, TfgPrimitiva* __restrict__ tris) {
    constexpr int kWords = (int)(sizeof(TfgPrimitiva) / 8);
    const int lane = threadIdx.x & 31;
    for (int base = (blockIdx.x * blockDim.x + threadIdx.x) & ~31; base < n; base += gridDim.x * blockDim.x) {
        const int i = base + lane;
        const bool tri = i < n && p[i].tipo == TFG_TRIANGULO;
        const uint32_t k = tri ? pos[i] - 1u : 0u;
        const uint32_t mask = __ballot_sync(0xFFFFFFFFu, tri);
        const unsigned long long* src = reinterpret_cast<const unsigned long long*>(p + base);
        if (mask == 0xFFFFFFFFu) {
            unsigned long long* dst =
                reinterpret_cast<unsigned long long*>(tris + __shfl_sync(0xFFFFFFFFu, k, 0));
#pragma unroll
            for (int w = 0; w < kWords; ++w) dst[32 * w + lane] = __ldg(&src[32 * w + lane]);
        } else {
            for (uint32_t m = mask; m; m &= m - 1u) {
                const int j = __ffs(m) - 1;
                unsigned long long* dst =
                    reinterpret_cast<unsigned long long*>(tris + __shfl_sync(0xFFFFFFFFu, k, j));
                if (lane < kWords) dst[lane] = __ldg(&src[kWords * j + lane]);
            }
        }
    }
}

__global__ void k_morton(const BNode* __restrict__ box, uint32_t n, const BuildWords* __restrict__ words,
                         uint32_t* __restrict__ code, uint32_t* __restrict__ idx) {
    float lo[3], inv[3];
    for (int a = 0; a < 3; ++a) {
        lo[a] = funkey(words->cb[a]);
        const float ext = funkey(words->cb[3 + a]) - lo[a];
        inv[a] = ext > 0.0f ? 1.0f / ext : 0.0f;
    }
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uint32_t q[3];
        for (int a = 0; a < 3; ++a) {
            const float c = (0.5f * (box[i].lo[a] + box[i].hi[a]) - lo[a]) * inv[a];
            q[a] = (uint32_t)fminf(fmaxf(c * 1024.0f, 0.0f), 1023.0f);
        }
        code[i] = (expand_bits(q[0]) << 2) | (expand_bits(q[1]) << 1) | expand_bits(q[2]);
        idx[i] = i;
    }
}

// Binary radix tree: internal nodes 0..n-2, leaf i (sorted position) is node
// n - 1 + i.  child[i] = (left, right); parent of every node.
__device__ __forceinline__ int delta_of(const uint32_t* code, int n, int i, int j) {
    if (j < 0 || j >= n) return -1;
    const uint32_t a = code[i], b = code[j];
    return a == b ? 32 + __clz((uint32_t)(i ^ j)) : __clz(a ^ b);
}

__global__ void k_radix_tree(const uint32_t* __restrict__ code, int n, int2* __restrict__ child,
                             int* __restrict__ parent) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n - 1; i += gridDim.x * blockDim.x) {
        const int d = (delta_of(code, n, i, i + 1) - delta_of(code, n, i, i - 1)) >= 0 ? 1 : -1;
        const int dmin = delta_of(code, n, i, i - d);
        int lmax = 2;
        while (delta_of(code, n, i, i + lmax * d) > dmin) lmax *= 2;
        int l = 0;
        for (int t = lmax / 2; t >= 1; t /= 2)
            if (delta_of(code, n, i, i + (l + t) * d) > dmin) l += t;
        const int j = i + l * d;
        const int dnode = delta_of(code, n, i, j);
        int s = 0;
        for (int t = (l + 1) / 2;; t = (t + 1) / 2) {
            if (delta_of(code, n, i, i + (s + t) * d) > dnode) s += t;
            if (t == 1) break;
        }
        const int gamma = i + s * d + min(d, 0);
        const int left = min(i, j) == gamma ? (n - 1 + gamma) : gamma;
        const int right = max(i, j) == gamma + 1 ? (n - 1 + gamma + 1) : gamma + 1;
        child[i] = make_int2(left, right);
        parent[left] = i;
        parent[right] = i;
    }
}

// The plan of a binary node from its area, triangle count and its children's
// costs (C(n, 1) = min(leaf, wide node); C(n, i) = min(C(n, i - 1), D(n, i));
// D(n, j) = min over k of C(left, k) + C(right, j - k)).
__device__ __forceinline__ void plan_node(Plan2& P, float area, int count, const float (&lc)[8], const float (&rc)[8]) {
    float dist[9];
    uint8_t split[9];
#pragma unroll
    for (int j = 2; j <= 8; ++j) {
        dist[j] = INFINITY;
        split[j] = 0;
#pragma unroll
        for (int k = 1; k < j; ++k) {
            const float c = lc[k - 1] + rc[j - k - 1];
            if (c < dist[j]) { dist[j] = c; split[j] = (uint8_t)k; }
        }
    }
    const float leaf = count <= kMaxLeaf ? area * (float)count * kCostWideTri : INFINITY;
    const float internal = dist[8] + area * kCostWideNode;
    P.split8 = split[8];
    if (leaf <= internal) { P.cost[0] = leaf; P.how[0] = kLeaf; }
    else { P.cost[0] = internal; P.how[0] = kInternal; }
#pragma unroll
    for (int i = 2; i <= 8; ++i) {
        if (dist[i] < P.cost[i - 2]) { P.cost[i - 1] = dist[i]; P.how[i - 1] = (uint8_t)(kSplit + split[i]); }
        else { P.cost[i - 1] = P.cost[i - 2]; P.how[i - 1] = kSame; }
    }
}

__device__ __forceinline__ bool is_leaf2(int node, int n) { return node >= n - 1; }

__device__ __forceinline__ BNode load_node(const BNode* b) {   // written by another thread of this kernel
    const float4* q = reinterpret_cast<const float4*>(b);
    const float4 x = __ldcg(q), y = __ldcg(q + 1);
    BNode r;
    r.lo[0] = x.x; r.lo[1] = x.y; r.lo[2] = x.z; r.count = __float_as_int(x.w);
    r.hi[0] = y.x; r.hi[1] = y.y; r.hi[2] = y.z; r.pad = 0.0f;
    return r;
}

// Boxes, counts and plans bottom-up.  A thread stops at the first node whose
// other child is not finished yet; the second thread to arrive continues, its
// own child's box and costs in registers, and reads only the sibling's.  The
// chain of ~20 such steps is latency (atomic, fence, sibling): 16-byte loads
// issued together and no plans stored for single triangles.
__global__ void __launch_bounds__(256) k_refit(const BNode* __restrict__ tbox, const uint32_t* __restrict__ sorted,
                                               int n, const int2* __restrict__ child, const int* __restrict__ parent,
                                               BNode* box, Plan2* plan, uint32_t* arrivals) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int node = n - 1 + i;
        BNode own = tbox[sorted[i]];
        box[node] = own;
        float cost[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) cost[k] = box_area(own) * 1.0f * kCostWideTri;
        while (node != 0) {
            const int p = parent[node];
            const int2 c = child[p];
            __threadfence();
            if (atomicAdd(&arrivals[p], 1u) == 0u) break;
            __threadfence();
            const bool left = c.x == node;
            const int sib = left ? c.y : c.x;
            const BNode o = load_node(&box[sib]);
            float oc[8];
            if (is_leaf2(sib, n)) {
                const float l = box_area(o) * 1.0f * kCostWideTri;
#pragma unroll
                for (int k = 0; k < 8; ++k) oc[k] = l;
            } else {
                const float4* q = reinterpret_cast<const float4*>(plan[sib].cost);
                const float4 x = __ldcg(q), y = __ldcg(q + 1);
                oc[0] = x.x; oc[1] = x.y; oc[2] = x.z; oc[3] = x.w;
                oc[4] = y.x; oc[5] = y.y; oc[6] = y.z; oc[7] = y.w;
            }
            BNode r;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                r.lo[k] = fminf(own.lo[k], o.lo[k]);
                r.hi[k] = fmaxf(own.hi[k], o.hi[k]);
            }
            r.count = own.count + o.count;
            r.pad = 0.0f;
            box[p] = r;
            float lc[8], rc[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) { lc[k] = left ? cost[k] : oc[k]; rc[k] = left ? oc[k] : cost[k]; }
            Plan2 P;
            plan_node(P, box_area(r), r.count, lc, rc);
#pragma unroll
            for (int k = 0; k < 7; ++k) P.pad[k] = 0;
            plan[p] = P;
#pragma unroll
            for (int k = 0; k < 8; ++k) cost[k] = P.cost[k];
            own = r;
            node = p;
        }
    }
}

struct WideArgs {
    const int2* child;
    const BNode* box;
    const Plan2* plan;
    const uint32_t* sorted;   // sorted position -> compacted triangle index
    int n;                    // triangles
    int level;
    const int2* q_in;         // (binary node, wide index)
    int2* q_out;
    BuildWords* words;
    uint32_t* nodes;          // 20 words per wide node
    uint32_t* tri_order;      // leaf order -> compacted triangle index
};

__device__ int gather_leaf_tris(const WideArgs& a, int node, uint32_t (&out)[kMaxLeaf]) {
    int stack[8], sp = 0, cnt = 0;
    stack[sp++] = node;
    while (sp > 0 && cnt < kMaxLeaf) {
        const int m = stack[--sp];
        if (is_leaf2(m, a.n)) {
            out[cnt++] = a.sorted[m - (a.n - 1)];
        } else {
            const int2 c = a.child[m];
            stack[sp++] = c.y;
            stack[sp++] = c.x;
        }
    }
    return cnt;
}

// 2^e as a double, e in [-1022, 1023].
__device__ __forceinline__ double pow2(int e) { return __hiloint2double((1023 + e) << 20, 0); }

// Exponent of the quantisation step along one axis: the smallest e >= -126
// with 255 * 2^e >= ext (0 extent: -126), at most 127.
__device__ __forceinline__ int grid_exponent(double ext) {
    int ex = -126;
    if (ext > 0.0) {
        ex = (int)ceil(log2(ext / 255.0));
        while (ldexp(255.0, ex) < ext) ++ex;
        ex = max(ex, -126);
    }
    return min(ex, 127);
}

// One wide node per eight lanes: the host builder's cost-optimal collapse
// (read from the plans), slot assignment and quantisation (cwbvh_build.cpp)
// on this level's queue.  A level's time is one node's latency while the
// levels are small, so a node's work is spread over its lanes: they hold its
// children left to right and open all open ones in each round (a thread per
// node walked the plan child by child, kept 64 double costs in local memory
// and took 51 us per level of an 81,920-triangle build).
constexpr int kWideThreads = 128;

__global__ void __launch_bounds__(kWideThreads) k_wide_level(WideArgs a) {
    __shared__ int4 s_item[kWideThreads / 8][8];       // (binary node, budget or lane, state, -)
    __shared__ __align__(16) uint32_t s_node[kWideThreads / 8][20];
    constexpr uint32_t kFull = 0xFFFFFFFFu;
    const uint32_t qn = a.words->level[a.level];
    const uint32_t lane = threadIdx.x & 31u, j = threadIdx.x & 7u, g = threadIdx.x >> 3, g0 = lane & 24u;
    const uint32_t stride = gridDim.x * (kWideThreads / 8);
    for (uint32_t base = blockIdx.x * (kWideThreads / 8) + (threadIdx.x >> 5) * 4u; base < qn; base += stride) {
        const bool act = base + (lane >> 3) < qn;
        int node2 = 0, widx = 0;
        if (act) { const int2 q = a.q_in[base + (lane >> 3)]; node2 = q.x; widx = q.y; }
        // ---- children: lane j holds the j-th from the left
        int item = -1, budget = 0, nk = 0;
        bool leaf = false, open = false;
        if (act) {
            if (is_leaf2(node2, a.n)) {
                nk = 1;
                if (j == 0) { item = node2; leaf = true; }
            } else {
                // (no split was finite over non-finite boxes: split8 = 0)
                const int k8 = a.plan[node2].split8 ? a.plan[node2].split8 : 4;
                const int2 c = a.child[node2];
                nk = 2;
                if (j < 2) { item = j == 0 ? c.x : c.y; budget = j == 0 ? k8 : 8 - k8; open = true; }
            }
        }
        while (__any_sync(kFull, open)) {
            bool split = false;
            int kl = 0;
            int2 c = make_int2(0, 0);
            if (open) {
                if (is_leaf2(item, a.n)) {
                    leaf = true;
                    open = false;
                } else {
                    const uint2 how = *reinterpret_cast<const uint2*>(a.plan[item].how);
                    c = a.child[item];
                    auto at = [&](int b) { return ((b < 4 ? how.x : how.y) >> (8 * (b & 3))) & 0xFFu; };
                    while (budget > 1 && at(budget - 1) == kSame) --budget;
                    const uint32_t h = at(budget - 1);
                    if (h == kLeaf || h == kInternal) {
                        leaf = h == kLeaf;
                        open = false;
                    } else {
                        split = true;
                        kl = (int)h - kSplit;
                    }
                }
            }
            const uint32_t sm = (__ballot_sync(kFull, split) >> g0) & 0xFFu;
            const int at = (int)j + __popc(sm & ((1u << j) - 1u));
            if ((int)j < nk) {
                s_item[g][at] = make_int4(split ? c.x : item, split ? kl : budget, (open ? 1 : 0) | (leaf ? 2 : 0), 0);
                if (split) s_item[g][at + 1] = make_int4(c.y, budget - kl, 1, 0);
            }
            nk += __popc(sm);
            __syncwarp();
            if ((int)j < nk) {
                const int4 v = s_item[g][j];
                item = v.x; budget = v.y; open = v.z & 1; leaf = (v.z & 2) != 0;
            }
            __syncwarp();
        }
        // ---- octant slots, greedy on dot(c_child - c_parent, dir_s): the
        // least cost, then the leftmost child, then the lowest slot
        const bool kid = act && (int)j < nk;
        BNode pb{}, cb{};
        if (act) pb = a.box[node2];
        if (kid) cb = a.box[item];
        double d[3];
#pragma unroll
        for (int k = 0; k < 3; ++k)
            d[k] = 0.5 * ((double)cb.lo[k] + (double)cb.hi[k]) - 0.5 * ((double)pb.lo[k] + (double)pb.hi[k]);
        uint32_t taken = 0;
        int slot = -1;
        while (__any_sync(kFull, kid && slot < 0)) {
            double best = INFINITY;
            int bs = -1;
            if (kid && slot < 0) {
#pragma unroll
                for (int s = 0; s < 8; ++s) {
                    const double c = d[0] * ((s & 4) ? -1.0 : 1.0) + d[1] * ((s & 2) ? -1.0 : 1.0) +
                                     d[2] * ((s & 1) ? -1.0 : 1.0);
                    if (!((taken >> s) & 1u) && (c < best || bs < 0)) { best = c; bs = s; }
                }
            }
            int bj = bs < 0 ? 8 : (int)j;
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) {
                const double ob = __shfl_xor_sync(kFull, best, o);
                const int oj = __shfl_xor_sync(kFull, bj, o), os = __shfl_xor_sync(kFull, bs, o);
                if (oj < 8 && (bj == 8 || ob < best || (ob == best && oj < bj))) { best = ob; bj = oj; bs = os; }
            }
            bj = __shfl_sync(kFull, bj, 0, 8);   // one lane's choice for the group, whatever the costs
            bs = __shfl_sync(kFull, bs, 0, 8);
            if (bj < 8) {
                taken |= 1u << bs;
                if (bj == (int)j) slot = bs;
            }
        }
        // ---- lane j takes the child in slot j
        s_item[g][j] = make_int4(-1, (int)j, 0, 0);
        __syncwarp();
        if (kid) s_item[g][slot] = make_int4(item, (int)j, leaf ? 2 : 0, 0);
        __syncwarp();
        const int4 mine = s_item[g][j];
        const bool has = mine.x >= 0;
        leaf = has && (mine.z & 2) != 0;
        const bool inner = has && !leaf;
        float lo[3], hi[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            lo[k] = __shfl_sync(kFull, cb.lo[k], mine.y, 8);
            hi[k] = __shfl_sync(kFull, cb.hi[k], mine.y, 8);
        }
        uint32_t tri[kMaxLeaf];
        const int cnt = leaf ? gather_leaf_tris(a, mine.x, tri) : 0;
        // ---- reserve the inner children's node block and the leaf triangles' block
        const uint32_t im = __ballot_sync(kFull, inner);
        int tsum = cnt;   // running triangle count over the warp's slots
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(kFull, tsum, o);
            if ((int)lane >= o) tsum += v;
        }
        const uint32_t ni = (uint32_t)__popc(im), nt = (uint32_t)__shfl_sync(kFull, tsum, 31);
        uint32_t r0 = 0, r1 = 0, r2 = 0;
        if (lane == 0) {
            if (ni) { r0 = atomicAdd(&a.words->next_node, ni); r2 = atomicAdd(&a.words->level[a.level + 1], ni); }
            if (nt) r1 = atomicAdd(&a.words->next_tri, nt);
        }
        r0 = __shfl_sync(kFull, r0, 0);
        r1 = __shfl_sync(kFull, r1, 0);
        r2 = __shfl_sync(kFull, r2, 0);
        const uint32_t gi = (im >> g0) & 0xFFu;                                   // the node's inner slots
        const uint32_t ibefore = (uint32_t)__popc(im & ((1u << g0) - 1u));        // inner children of earlier nodes
        const uint32_t rank = (uint32_t)__popc(gi & ((1u << j) - 1u));
        const uint32_t tfirst = (uint32_t)(__shfl_sync(kFull, tsum, (int)g0) - __shfl_sync(kFull, cnt, (int)g0));
        const uint32_t gtris = (uint32_t)__shfl_sync(kFull, tsum, (int)g0 + 7) - tfirst;
        const uint32_t toff = (uint32_t)(tsum - cnt) - tfirst;
        const uint32_t child_base = gi ? r0 + ibefore : 0u, tri_base = gtris ? r1 + tfirst : 0u;
        // ---- quantisation and the node's 80 bytes
        uint8_t* nb = reinterpret_cast<uint8_t*>(s_node[g]);
        const int axis = j < 2 ? (int)j : 2;
        const int ej = grid_exponent((double)(axis == 0 ? pb.hi[0] : axis == 1 ? pb.hi[1] : pb.hi[2]) -
                                     (double)(axis == 0 ? pb.lo[0] : axis == 1 ? pb.lo[1] : pb.lo[2]));
        int e[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            e[k] = __shfl_sync(kFull, ej, k, 8);
            const double inv = pow2(-e[k]);
            const double ql = floor(((double)lo[k] - (double)pb.lo[k]) * inv);
            const double qh = ceil(((double)hi[k] - (double)pb.lo[k]) * inv);
            nb[32 + 8 * k + j] = has ? (uint8_t)fmin(fmax(ql, 0.0), 255.0) : (uint8_t)0;
            nb[56 + 8 * k + j] = has ? (uint8_t)fmin(fmax(qh, 0.0), 255.0) : (uint8_t)0;
        }
        nb[24 + j] = leaf ? (uint8_t)((((1u << cnt) - 1u) << 5) | toff) : inner ? (uint8_t)((1u << 5) | (24u + j)) : (uint8_t)0;
        if (j == 0) {
            uint32_t* w = s_node[g];
            w[0] = __float_as_uint(pb.lo[0]); w[1] = __float_as_uint(pb.lo[1]); w[2] = __float_as_uint(pb.lo[2]);
            w[3] = (uint32_t)(uint8_t)(int8_t)e[0] | ((uint32_t)(uint8_t)(int8_t)e[1] << 8) |
                   ((uint32_t)(uint8_t)(int8_t)e[2] << 16) | (gi << 24);
            w[4] = child_base;
            w[5] = 4u * tri_base;
        }
        if (leaf)
            for (int k = 0; k < cnt; ++k) a.tri_order[tri_base + toff + (uint32_t)k] = tri[k];
        if (inner) a.q_out[r2 + ibefore + rank] = make_int2(mine.x, (int)(child_base + rank));
        __syncwarp();
        if (act && j < 5)
            reinterpret_cast<uint4*>(a.nodes + 20 * (size_t)widx)[j] = reinterpret_cast<const uint4*>(s_node[g])[j];
        __syncwarp();
    }
}

// Both triangle layouts in leaf order (the host builder's formulas).
__global__ void k_emit_tris(const float* __restrict__ verts, const uint32_t* __restrict__ order, uint32_t nt,
                            float* __restrict__ tris_ref, float* __restrict__ tris_wt) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < nt; k += gridDim.x * blockDim.x) {
        const uint32_t t = order[k];
        const float* tv = &verts[9 * (size_t)t];
        float4* W = reinterpret_cast<float4*>(tris_wt) + 3 * (size_t)k;
        W[0] = make_float4(tv[0], tv[1], tv[2], __uint_as_float(t));
        W[1] = make_float4(tv[3], tv[4], tv[5], 0.0f);
        W[2] = make_float4(tv[6], tv[7], tv[8], 0.0f);
        const double v0[3] = {tv[0], tv[1], tv[2]};
        const double e1[3] = {tv[3] - v0[0], tv[4] - v0[1], tv[5] - v0[2]};
        const double e2[3] = {tv[6] - v0[0], tv[7] - v0[1], tv[8] - v0[2]};
        auto cross = [](const double* x, const double* y, double* r) {
            r[0] = x[1] * y[2] - x[2] * y[1];
            r[1] = x[2] * y[0] - x[0] * y[2];
            r[2] = x[0] * y[1] - x[1] * y[0];
        };
        double nrm[3], r0[3], r1[3];
        cross(e1, e2, nrm);
        const double n2 = nrm[0] * nrm[0] + nrm[1] * nrm[1] + nrm[2] * nrm[2];
        float4* R = reinterpret_cast<float4*>(tris_ref) + 4 * (size_t)k;
        if (!(n2 > 0.0) || !isfinite(n2)) {
            R[0] = R[1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            R[2] = make_float4(0.0f, 0.0f, 0.0f, 1.0f);
        } else {
            cross(e2, nrm, r0);
            cross(nrm, e1, r1);
            const double inv = 1.0 / n2;
            double rows[3][3];
            for (int c = 0; c < 3; ++c) { rows[0][c] = r0[c] * inv; rows[1][c] = r1[c] * inv; rows[2][c] = nrm[c] * inv; }
            for (int r = 0; r < 3; ++r) {
                const double wv = -(rows[r][0] * v0[0] + rows[r][1] * v0[1] + rows[r][2] * v0[2]);
                R[r] = make_float4((float)rows[r][0], (float)rows[r][1], (float)rows[r][2], (float)wv);
            }
        }
        R[3] = make_float4(0.0f, 0.0f, 0.0f, __uint_as_float(t));
    }
}

// Pool of each device that builds' scratch blocks come from: stream-ordered,
// keeping at most kPoolKeep bytes between builds.  A pool gives what it holds
// above that back at the next synchronisation after the memory was freed, so a
// build frees its scratch before it synchronises for the last time (freed after
// it, the 0.5 GB of a 2 M triangle build stayed until the program synchronised
// again).  One block per build,
// so builds on several threads or streams never share memory.
constexpr uint64_t kPoolKeep = 128ull << 20;
std::mutex g_pool_mutex;
cudaMemPool_t g_pool[kMaxDevices] = {nullptr};

cudaError_t build_pool(int dev, cudaMemPool_t* out) {
    std::lock_guard<std::mutex> lk(g_pool_mutex);
    if (!g_pool[dev]) {
        cudaMemPoolProps props;
        std::memset(&props, 0, sizeof(props));
        props.allocType = cudaMemAllocationTypePinned;
        props.handleTypes = cudaMemHandleTypeNone;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool = nullptr;
        cudaError_t e = cudaMemPoolCreate(&pool, &props);
        uint64_t keep = kPoolKeep;
        if (e == cudaSuccess) e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
        if (e != cudaSuccess) {
            if (pool) cudaMemPoolDestroy(pool);
            return e;
        }
        g_pool[dev] = pool;
    }
    *out = g_pool[dev];
    return cudaSuccess;
}

// One scratch block, carved into 256-byte aligned arrays; freed in stream
// order, on an early exit with a synchronisation of its own.
struct Scratch {
    cudaStream_t s;
    uint8_t* base = nullptr;
    size_t used = 0;
    explicit Scratch(cudaStream_t st) : s(st) {}
    cudaError_t reserve(cudaMemPool_t pool, size_t bytes) {
        return cudaMallocFromPoolAsync((void**)&base, bytes, pool, s);
    }
    static size_t pad(size_t bytes) { return (bytes + 255) & ~size_t(255); }
    template <typename T>
    T* get(size_t count) {
        T* q = reinterpret_cast<T*>(base + used);
        used += pad(count * sizeof(T));
        return q;
    }
    cudaError_t release() {
        uint8_t* b = base;
        base = nullptr;
        return b ? cudaFreeAsync(b, s) : cudaSuccess;
    }
    ~Scratch() {
        if (!base) return;
        release();
        cudaStreamSynchronize(s);
    }
};

}  // namespace
}  // namespace tfg

extern "C" int tfgTinyBVHConstruirGPU(const TfgPrimitiva* d_prims, int32_t n, TfgTinyBVH* out, void* stream) {
    using namespace tfg;
    if (!out) return fail(TFG_E_INVALID, "tfgTinyBVHConstruirGPU: out is null");
    std::memset(out, 0, sizeof(*out));
    if (n < 0 || (n > 0 && !d_prims)) return fail(TFG_E_INVALID, "tfgTinyBVHConstruirGPU: bad primitive array");
    if (n == 0) return ok();
    cudaStream_t s = (cudaStream_t)stream;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return fail((int)e, cudaGetErrorString(e));
    if (int rc = require_sm100(dev)) return rc;
    auto bail = [&](cudaError_t err) {
        tfgTinyBVHLiberar(out);
        return fail((int)err, std::string("tfgTinyBVHConstruirGPU: ") + cudaGetErrorString(err));
    };
    cudaMemPool_t pool = nullptr;
    e = build_pool(dev, &pool);
    if (e != cudaSuccess) return bail(e);
    // how many triangles there are: the last value of a running count
    const auto flags = thrust::make_transform_iterator(d_prims, IsTriangle{});
    Scratch scan(s);
    size_t scan_bytes = 0;
    e = cub::DeviceScan::InclusiveSum(nullptr, scan_bytes, flags, (uint32_t*)nullptr, n, s);
    if (e == cudaSuccess) e = scan.reserve(pool, Scratch::pad((size_t)n * 4) + Scratch::pad(scan_bytes));
    if (e != cudaSuccess) return bail(e);
    uint32_t* pos = scan.get<uint32_t>(n);
    void* scan_tmp = scan.get<uint8_t>(scan_bytes);
    uint32_t nt = 0;
    e = cub::DeviceScan::InclusiveSum(scan_tmp, scan_bytes, flags, pos, n, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(&nt, pos + n - 1, 4, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return bail(e);
    if (nt == 0) return ok();   // no triangles: an empty BVH, as the host path
    if (nt > (1u << 29)) return fail(TFG_E_INVALID, "tfgTinyBVHConstruirGPU: too many triangles");

    const size_t nn = 2 * (size_t)nt - 1;
    size_t sort_bytes = 0;
    e = cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, (uint32_t*)nullptr, (uint32_t*)nullptr,
                                        (uint32_t*)nullptr, (uint32_t*)nullptr, (int)nt, 0, 30, s);
    if (e != cudaSuccess) return bail(e);
    Scratch sc(s);
    const size_t sizes[] = {9 * (size_t)nt * 4, (size_t)nt * sizeof(BNode), sizeof(BuildWords), (size_t)nt * 4,
                            (size_t)nt * 4, (size_t)nt * 4, (size_t)nt * 4, (size_t)nt * sizeof(int2), nn * 4,
                            nn * sizeof(BNode), (size_t)nt * sizeof(Plan2), (size_t)nt * 4,
                            ((size_t)nt + 1) * sizeof(int2), ((size_t)nt + 1) * sizeof(int2),
                            80 * ((size_t)nt + 1), (size_t)nt * 4, sort_bytes};
    size_t total = 0;
    for (size_t b : sizes) total += Scratch::pad(b);
    e = sc.reserve(pool, total);
    if (e != cudaSuccess) return bail(e);
    float* verts = sc.get<float>(9 * (size_t)nt);
    BNode* tbox = sc.get<BNode>(nt);
    BuildWords* words = sc.get<BuildWords>(1);
    uint32_t* code = sc.get<uint32_t>(nt);
    uint32_t* code_s = sc.get<uint32_t>(nt);
    uint32_t* idx = sc.get<uint32_t>(nt);
    uint32_t* idx_s = sc.get<uint32_t>(nt);
    int2* child = sc.get<int2>(nt);
    int* parent = sc.get<int>(nn);
    BNode* box = sc.get<BNode>(nn);
    Plan2* plan = sc.get<Plan2>(nt);
    uint32_t* arrivals = sc.get<uint32_t>(nt);
    int2* q[2];
    q[0] = sc.get<int2>((size_t)nt + 1);
    q[1] = sc.get<int2>((size_t)nt + 1);
    uint32_t* nodes = sc.get<uint32_t>(20 * ((size_t)nt + 1));
    uint32_t* tri_order = sc.get<uint32_t>(nt);
    void* sort_tmp = sc.get<uint8_t>(sort_bytes);

    const uint32_t blocks = std::min<uint32_t>(((uint32_t)n + 255) / 256, 148u * 8u);
    const uint32_t tb = std::min<uint32_t>((nt + 255) / 256, 148u * 8u);
    k_build_init<<<tb, 256, 0, s>>>(words, q[0], arrivals, nt);
    k_compact<<<blocks, 256, 0, s>>>(d_prims, n, pos, verts, tbox, words);
    k_morton<<<tb, 256, 0, s>>>(tbox, nt, words, code, idx);
    e = cub::DeviceRadixSort::SortPairs(sort_tmp, sort_bytes, code, code_s, idx, idx_s, (int)nt, 0, 30, s);
    if (e != cudaSuccess) return bail(e);
    if (nt > 1) k_radix_tree<<<tb, 256, 0, s>>>(code_s, (int)nt, child, parent);
    k_refit<<<tb, 256, 0, s>>>(tbox, idx_s, (int)nt, child, parent, box, plan, arrivals);
    // Level-by-level collapse, kLevelBatch levels per host read.
    constexpr int kLevelBatch = 8;
    BuildWords hw;
    WideArgs wa;
    wa.child = child; wa.box = box; wa.plan = plan; wa.sorted = idx_s; wa.n = (int)nt;
    wa.words = words; wa.nodes = nodes; wa.tri_order = tri_order;
    const uint32_t per_block = kWideThreads / 8;
    const uint32_t wb = std::min<uint32_t>((nt + per_block - 1) / per_block, 148u * 8u);
    const size_t pb = Scratch::pad((size_t)nt * sizeof(TfgPrimitiva)), rb = Scratch::pad((size_t)nt * 64),
                 wtb = Scratch::pad((size_t)nt * 48), node_room = nt / 8 + 16;
    uint8_t* block = nullptr;
    int depth = 0;
    do {
        for (int k = 0; k < kLevelBatch; ++k, ++depth) {
            wa.level = depth; wa.q_in = q[depth & 1]; wa.q_out = q[(depth + 1) & 1];
            k_wide_level<<<wb, kWideThreads, 0, s>>>(wa);
        }
        if (!block) {
            // The result, one allocation, made while the GPU works: the
            // triangle arrays and room for the nodes (trees take 0.11 nodes
            // per triangle; one that needs more gets them on their own).
            e = cudaMalloc((void**)&block, pb + rb + wtb + node_room * 80);
            if (e != cudaSuccess) return bail(e);
            out->d_primitivas = reinterpret_cast<TfgPrimitiva*>(block);
            out->num_primitivas = nt;
            out->ref.d_tris = reinterpret_cast<float*>(block + pb);
            out->d_tris_wt = reinterpret_cast<float*>(block + pb + rb);
            bvh_register_block(block);
        }
        e = cudaMemcpyAsync(&hw, words, sizeof(hw), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) return bail(e);
    } while (hw.level[depth] != 0 && depth < 64);
    while (depth > 0 && hw.level[depth - 1] == 0) --depth;
    if (hw.level[64] != 0) {   // a valid tree is far shallower
        tfgTinyBVHLiberar(out);
        return fail(TFG_E_BUILD, "tfgTinyBVHConstruirGPU: tree deeper than 64 levels");
    }
    if (hw.next_tri != nt) {
        tfgTinyBVHLiberar(out);
        return fail(TFG_E_BUILD, "tfgTinyBVHConstruirGPU: leaves do not cover every triangle");
    }
    const uint32_t num_nodes = hw.next_node;
    k_emit_tris<<<tb, 256, 0, s>>>(verts, tri_order, nt, out->ref.d_tris, out->d_tris_wt);
    k_copy_prims<<<blocks, 256, 0, s>>>(d_prims, n, pos, out->d_primitivas);
    if (num_nodes <= node_room) out->ref.d_nodos = reinterpret_cast<float*>(block + pb + rb + wtb);
    else e = cudaMalloc((void**)&out->ref.d_nodos, (size_t)num_nodes * 80);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(out->ref.d_nodos, nodes, (size_t)num_nodes * 80, cudaMemcpyDeviceToDevice, s);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess) e = scan.release();
    if (e == cudaSuccess) e = sc.release();
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return bail(e);
    out->ref.num_nodos = num_nodes;
    out->ref.num_tris = nt;
    out->max_depth = (uint32_t)depth;
    return ok();
}
