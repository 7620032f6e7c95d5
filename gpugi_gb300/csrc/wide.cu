// Four-wide copy of an axis-aligned-box hierarchy for the ray walkers.
//
// The binary escape tree stays the scene's hierarchy (export, importance,
// oracle parity); this is a second, derived layout of the same tree in which
// every second level is left out: a wide node holds the boxes of the (two to
// four) grandchildren, or children that are leaves, of a binary node at even
// depth, in preorder, as structure-of-arrays in one 128-B line:
//   {lo.x[4]} {hi.x[4]} {lo.y[4]} {hi.y[4]} {lo.z[4]} {hi.z[4]} {ref[4]} {unused}
// ref: a wide node index, or the binary tree's leaf word (LEAF_FLAG | count |
// block), or kWideEmpty. Boxes are the binary nodes' own floats.
//
// Which walks may use it (wide_walks, trace.cuh) rests on the tree being what
// bvhmake and the LBVH builder write; gpugi_scene_upload accepts any forward
// escape graph, so it is checked here, edge by edge, on the device: every
// inner node has exactly two children, the right one is the left one's escape
// and shares its parent's escape, no node has two parents, and every child's
// box lies inside its parent's (and is not empty or NaN). A scene that fails
// any of it keeps the binary walkers.
//
// Bound by launch latency for small trees (5 us a kernel at 34k nodes) and by
// the parent climb of k_wide_mark for large ones; once per scene.
#include <cub/cub.cuh>

#include "ctx.cuh"

namespace gpugi {
namespace {

constexpr uint32_t kNoParent = 0xFFFFFFFFu;

GPUGI_D uint32_t child_word(const float4* nodes, uint32_t i) { return __float_as_uint(__ldg(nodes + 2 * (size_t)i).w); }
GPUGI_D uint32_t escape_word(const float4* nodes, uint32_t i) {
    return __float_as_uint(__ldg(nodes + 2 * (size_t)i + 1).w);
}

// parent[] of every child (kNoParent before), and the structure checks (*bad
// becomes 0 where one fails).
__global__ void k_wide_parents(const float4* __restrict__ nodes, uint32_t n, uint32_t* parent, uint32_t* bad) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t c = child_word(nodes, i);
    if (c & LEAF_FLAG) return;
    const uint32_t r = c < n ? escape_word(nodes, c) : 0u;
    bool ok = c > i && c < n && r > c && r < n && escape_word(nodes, r) == escape_word(nodes, i);
    if (ok) ok = atomicExch(parent + c, i) == kNoParent && atomicExch(parent + r, i) == kNoParent;
    if (!ok || (i == 0 && escape_word(nodes, 0) != 0u)) *bad = 0u;
}

// flag[i] = 1 for inner nodes at even depth below the root, flag[n] = 0;
// *minNotDepth = ~(depth of the deepest inner node). Parents have smaller
// indexes than their children, so the climb ends.
__global__ void k_wide_mark(const float4* __restrict__ nodes, uint32_t n, const uint32_t* __restrict__ parent,
                            uint32_t* __restrict__ flag, uint32_t* minNotDepth) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t depth = 0;
    if (i < n) {
        bool mark = false;
        if (!(child_word(nodes, i) & LEAF_FLAG)) {
            uint32_t v = i;
            while (v != 0 && parent[v] < v) {
                v = parent[v];
                ++depth;
            }
            mark = v == 0 && (depth & 1u) == 0;
            if (v != 0) depth = 0;
        }
        flag[i] = mark ? 1u : 0u;
    } else if (i == n) {
        flag[n] = 0u;
    }
    depth = __reduce_max_sync(0xffffffffu, depth);
    if ((threadIdx.x & 31u) == 0 && depth) atomicMin(minNotDepth, ~depth);
}

__global__ void k_wide_fill(const float4* __restrict__ nodes, uint32_t n, const uint32_t* __restrict__ flag,
                            const uint32_t* __restrict__ index, uint32_t capacity, float4* __restrict__ wide,
                            uint32_t* bad) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || !flag[i] || index[i] >= capacity) return;
    uint32_t kid[4], count = 0;
    bool ok = true;
    auto inside = [&](uint32_t outer, uint32_t inner) {
        const float4 a = __ldg(nodes + 2 * (size_t)outer), b = __ldg(nodes + 2 * (size_t)outer + 1);
        const float4 c = __ldg(nodes + 2 * (size_t)inner), d = __ldg(nodes + 2 * (size_t)inner + 1);
        return a.x <= c.x && a.y <= c.y && a.z <= c.z && d.x <= b.x && d.y <= b.y && d.z <= b.z && c.x <= d.x &&
               c.y <= d.y && c.z <= d.z;
    };
    auto kids = [&](uint32_t p, uint32_t& l, uint32_t& r) {
        l = child_word(nodes, p);
        r = l < n ? escape_word(nodes, l) : n;
        if (l >= n || r >= n) return false;
        return inside(p, l) && inside(p, r);
    };
    uint32_t c[2];
    ok = kids(i, c[0], c[1]);
    for (int s = 0; s < 2 && ok; ++s) {
        if (child_word(nodes, c[s]) & LEAF_FLAG) {
            kid[count++] = c[s];
        } else {
            ok = kids(c[s], kid[count], kid[count + 1]);
            count += 2;
        }
    }
    if (!ok) {
        *bad = 0u;
        return;
    }
    float* w = reinterpret_cast<float*>(wide + 8 * (size_t)index[i]);
    for (uint32_t k = 0; k < 4; ++k) {
        uint32_t ref = kWideEmpty;
        float4 a = make_float4(0, 0, 0, 0), b = a;
        if (k < count) {
            a = __ldg(nodes + 2 * (size_t)kid[k]);
            b = __ldg(nodes + 2 * (size_t)kid[k] + 1);
            ref = __float_as_uint(a.w);
            if (!(ref & LEAF_FLAG)) {
                if (!flag[kid[k]]) *bad = 0u;
                ref = index[kid[k]];
            }
        }
        w[k] = a.x, w[4 + k] = b.x;
        w[8 + k] = a.y, w[12 + k] = b.y;
        w[16 + k] = a.z, w[20 + k] = b.z;
        w[24 + k] = __uint_as_float(ref);
        w[28 + k] = 0.0f;
    }
}

}  // namespace

gpugi_status build_wide(gpugi_ctx* ctx, gpugi_scene* sc) {
    sc->dev.wide = nullptr;
    sc->dev.numWide = 0;
    const uint32_t n = sc->dev.numNodes;
    if (sc->dev.boundsKind != GPUGI_BOUNDS_AABB || sc->dev.topNodes || n < 3) return GPUGI_OK;
    cudaStream_t st = ctx->stream;
    size_t scanBytes = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, scanBytes, (uint32_t*)nullptr, (uint32_t*)nullptr, (int)n + 1, st);
    // scratch in the context's staging buffer (kept between calls; every user of it finishes before it
    // returns): parent and {checks passed, ~depth}, flag, index (the node count at [n]), scan storage
    const size_t col = (4 * (size_t)n + 16 + 255) & ~size_t(255);
    if (gpugi_status gs = ensure_stage(ctx, 3 * col + scanBytes)) {
        cudaGetLastError();
        return gs == GPUGI_ERROR_OUT_OF_MEMORY ? GPUGI_OK : gs;  // the binary walkers need no extra memory
    }
    char* scratch = static_cast<char*>(ctx->stageDev);
    uint32_t* parent = reinterpret_cast<uint32_t*>(scratch);
    uint32_t* word = parent + n;
    uint32_t* flag = reinterpret_cast<uint32_t*>(scratch + col);
    uint32_t* index = reinterpret_cast<uint32_t*>(scratch + 2 * col);
    const unsigned grid = n / 256 + 1;  // covers [0, n]
    GPUGI_CUDA_TRY(ctx, cudaMemsetAsync(parent, 0xFF, 4 * ((size_t)n + 2), st));
    k_wide_parents<<<grid, 256, 0, st>>>(sc->dev.nodes, n, parent, word);
    k_wide_mark<<<grid, 256, 0, st>>>(sc->dev.nodes, n, parent, flag, word + 1);
    GPUGI_CUDA_TRY(ctx, cub::DeviceScan::ExclusiveSum(scratch + 3 * col, scanBytes, flag, index, (int)n + 1, st));
    // At most every inner node is a wide one: small trees allocate for that (64 B a node), so that the
    // host waits once; large ones read the count first.
    uint32_t count = (n - 1) / 2;
    if (n > (1u << 20)) {
        GPUGI_CUDA_TRY(ctx, cudaMemcpyAsync(&count, index + n, 4, cudaMemcpyDeviceToHost, st));
        GPUGI_CUDA_TRY(ctx, cudaStreamSynchronize(st));
        if (count > (n - 1) / 2) return GPUGI_OK;
    }
    if (count == 0) return GPUGI_OK;
    float4* wide = nullptr;
    if (cudaMalloc(&wide, 128 * (size_t)count) != cudaSuccess) {
        cudaGetLastError();
        return GPUGI_OK;
    }
    sc->allocations.push_back(wide);
    k_wide_fill<<<grid, 256, 0, st>>>(sc->dev.nodes, n, flag, index, count, wide, word);
    GPUGI_CUDA_TRY(ctx, cudaGetLastError());
    uint32_t got[3];
    GPUGI_CUDA_TRY(ctx, cudaMemcpyAsync(got, word, 8, cudaMemcpyDeviceToHost, st));
    GPUGI_CUDA_TRY(ctx, cudaMemcpyAsync(got + 2, index + n, 4, cudaMemcpyDeviceToHost, st));
    GPUGI_CUDA_TRY(ctx, cudaStreamSynchronize(st));
    // a walk's stack holds at most three entries per wide level, and its node offsets are 32-bit bytes
    const bool fits = 3 * (~got[1] / 2 + 1) <= kWideStack && got[2] < (1u << 25);
    if (got[0] == 0 || !fits || got[2] == 0 || got[2] > count) return GPUGI_OK;
    sc->wide = sc->dev.wide = wide;
    sc->dev.numWide = got[2];
    return GPUGI_OK;
}

}  // namespace gpugi
